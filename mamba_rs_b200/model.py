"""Host-side mirror of the reference's Mamba-1 engines on top of the C ABI.

The reference's engines are per-layer launch sequences around the scan
(``GpuMambaBackbone::prefill_sequence_mixed`` / ``step``,
src/mamba_ssm/gpu/inference.rs:1515-1855, prefill.rs:676-961; ``MambaTrainer``,
src/mamba_ssm/gpu/trainer.rs:437-481, forward_mixed.rs:433-758,
backward_mixed.rs:83-782).  This module keeps their method names and argument
meaning and issues the same sequence with this library's fused entry points:

    residual+RMSNorm | GEMM in_proj | conv1d+SiLU | GEMM x_proj | GEMM dt_proj |
    scan (softplus, D skip, SiLU(z) gate fused) | GEMM out_proj | (residual add fused
    into the next layer's norm)

The dense projections stay library GEMMs (``torch.matmul`` -> cuBLAS), as they are
cuBLAS calls in the reference: they are not part of the scan path.  Parameters and
their gradients live in flat f32 arenas (the reference's ``GpuMambaGrads.flat``,
src/mamba_ssm/gpu/weights.rs:487-560) with a compute-dtype copy beside the master,
so the data-parallel all-reduce and AdamW are one call each over the arena.
torch supplies device memory, streams and the process group, nothing else.
"""
from __future__ import annotations

import ctypes as C
import math
import weakref
from dataclasses import dataclass

import torch

from . import ffi, ops
from .parallel import BucketedGradReducer

__all__ = ["MambaConfig", "MambaWeights", "GpuMambaBackbone", "GpuMambaLM", "MambaLMTrainer"]


@dataclass
class MambaConfig:
    """src/config.rs:57-101."""
    d_model: int
    n_layers: int
    d_state: int = 16
    d_conv: int = 4
    expand: int = 2
    rms_norm_eps: float = 1e-5
    dt_rank: int | None = None

    def __post_init__(self):
        if self.dt_rank is None:
            self.dt_rank = (self.d_model + 15) // 16
        if not (1 <= self.d_conv <= 8):
            raise ValueError("d_conv must be 1..8")
        if not (1 <= self.d_state <= 256):
            raise ValueError("d_state must be 1..256")

    @property
    def d_inner(self):
        return self.expand * self.d_model

    @property
    def xdbl_dim(self):
        return self.dt_rank + 2 * self.d_state


_LAYER_FIELDS = ("norm_w", "in_proj_w", "conv_w", "conv_b", "x_proj_w", "dt_proj_w", "dt_proj_b", "a_log", "d_param",
                 "out_proj_w")


class MambaWeights:
    """Flat f32 master arena + compute-dtype copy, with named views per layer
    (src/weights.rs:8-65).  GEMM weights are [in, out] row-major, as in the reference."""

    def __init__(self, cfg: MambaConfig, device, dtype=torch.bfloat16, vocab: int | None = None):
        self.cfg, self.dtype, self.vocab = cfg, dtype, vocab
        dm, di, N, K, dr, xd = cfg.d_model, cfg.d_inner, cfg.d_state, cfg.d_conv, cfg.dt_rank, cfg.xdbl_dim
        self.shapes = dict(norm_w=(dm,), in_proj_w=(dm, 2 * di), conv_w=(di, K), conv_b=(di,), x_proj_w=(di, xd),
                           dt_proj_w=(dr, di), dt_proj_b=(di,), a_log=(di, N), d_param=(di,), out_proj_w=(di, dm))
        per_layer = sum(math.prod(s) for s in self.shapes.values())
        self.layer_size = (per_layer + 63) // 64 * 64  # buckets start on 256-byte boundaries
        extra = dm + (vocab * dm if vocab else 0)
        self.n = cfg.n_layers * self.layer_size + extra
        self.master = torch.zeros(self.n, device=device)
        device = self.device = self.master.device  # with its index, also where `device` is a name or has none
        self.grad = torch.zeros(self.n, device=device)
        self.lp = torch.zeros(self.n, device=device, dtype=dtype) if dtype != torch.float32 else self.master
        self._a_neg_all = torch.empty(cfg.n_layers, di, N, device=device)
        self.a_neg = list(self._a_neg_all)
        self._view_cache = {}

    # ---- views ----
    def _views(self, flat, l):
        o = l * self.layer_size
        out = {}
        for k in _LAYER_FIELDS:
            n = math.prod(self.shapes[k])
            out[k] = flat[o:o + n].view(self.shapes[k])
            o += n
        return out

    def _cached(self, key, flat, make):
        """Views of an arena are made once and kept while the arena is the same tensor."""
        got = self._view_cache.get(key)
        if got is None or got[0] is not flat:
            got = self._view_cache[key] = (flat, make())
        return got[1]

    def layer(self, l, which="lp"):
        flat = getattr(self, which)
        return self._cached((which, l), flat, lambda: self._views(flat, l))

    def tail(self, which="lp"):
        flat = getattr(self, which)
        return self._cached((which, "tail"), flat, lambda: self._tail_views(flat))

    def _tail_views(self, flat):
        o = self.cfg.n_layers * self.layer_size
        dm = self.cfg.d_model
        out = dict(norm_f=flat[o:o + dm])
        if self.vocab:
            out["embedding"] = flat[o + dm:o + dm + self.vocab * dm].view(self.vocab, dm)
        return out

    def bucket_bounds(self):
        """One gradient bucket per layer, then the tail (final norm, embedding)."""
        b = [(l * self.layer_size, (l + 1) * self.layer_size) for l in range(self.cfg.n_layers)]
        b.append((self.cfg.n_layers * self.layer_size, self.n))
        return b

    def refresh(self):
        """master -> compute copy, and a_neg = -exp(a_log) (trainer.rs:78-111)."""
        if self.lp is not self.master:
            self.lp.copy_(self.master)
        self.refresh_a_neg()

    def refresh_a_neg(self):
        """a_neg = -exp(a_log) of every layer, over the whole arena at once (unless a layer's tensor
        was replaced)."""
        whole = all(t.data_ptr() == self._a_neg_all[l].data_ptr() for l, t in enumerate(self.a_neg))
        if whole:
            a = self.layer(0, "master")["a_log"]
            logs = torch.as_strided(self.master, self._a_neg_all.shape, (self.layer_size, *a.stride()), a.storage_offset())
            torch.exp(logs, out=self._a_neg_all).neg_()
        else:
            for l in range(self.cfg.n_layers):
                torch.exp(self.layer(l, "master")["a_log"], out=self.a_neg[l]).neg_()

    def init_random(self, seed: int):
        """MambaWeights::init (src/weights.rs:107-160): Kaiming-uniform projections,
        A_log = ln(1..N), dt bias = inverse softplus of log-uniform dt in [1e-3, 1e-1], D = 1,
        norm weights 1 (the distributions; this generator is torch's, not the reference's LCG)."""
        g = torch.Generator(device=self.device).manual_seed(seed)
        cfg = self.cfg

        def kaiming(t, fan_in):
            bound = math.sqrt(3.0 / fan_in)
            t.copy_((torch.rand(t.shape, device=self.device, generator=g) * 2 - 1) * bound)

        for l in range(cfg.n_layers):
            v = self.layer(l, "master")
            v["norm_w"].fill_(1.0)
            kaiming(v["in_proj_w"], cfg.d_model)
            kaiming(v["conv_w"], cfg.d_conv)
            v["conv_b"].zero_()
            kaiming(v["x_proj_w"], cfg.d_inner)
            kaiming(v["dt_proj_w"], cfg.dt_rank)
            dt = torch.exp(torch.rand(cfg.d_inner, device=self.device, generator=g) *
                           (math.log(1e-1) - math.log(1e-3)) + math.log(1e-3))
            v["dt_proj_b"].copy_(dt + torch.log(-torch.expm1(-dt)))  # inverse softplus
            v["a_log"].copy_(torch.log(torch.arange(1, cfg.d_state + 1, device=self.device).float()).expand_as(v["a_log"]))
            v["d_param"].fill_(1.0)
            kaiming(v["out_proj_w"], cfg.d_inner)
        t = self.tail("master")
        t["norm_f"].fill_(1.0)
        if self.vocab:
            t["embedding"].copy_(torch.randn(t["embedding"].shape, device=self.device, generator=g) * 0.02)
        self.refresh()
        return self

    def load_layers(self, layers, norm_f):
        """Copies named numpy / tensor arrays (same field names) into the master arena."""
        for l, src in enumerate(layers):
            v = self.layer(l, "master")
            for k in _LAYER_FIELDS:
                v[k].copy_(torch.as_tensor(src[k], dtype=torch.float32).reshape(self.shapes[k]))
        self.tail("master")["norm_f"].copy_(torch.as_tensor(norm_f, dtype=torch.float32))
        self.refresh()
        return self


def _capturing(t):
    """Whether the current stream of t's device is being captured.  What is made then (a zeroed workspace, a
    row of ones) is filled by the graph's replays alone, so no later call may be given it: plans made
    inside a capture serve that call and go."""
    if not t.is_cuda:
        return False
    with ops._on(t.device):
        return torch.cuda.is_current_stream_capturing()


class _Lent:
    """Buffers that a plan keeps between calls.  Where a call runs on another stream than the one they were
    made on, the allocator is told, so that a plan which is dropped does not hand memory on that the call
    still reads."""

    def __init__(self, *tensors):
        self.tensors, self.dev = tensors, tensors[0].device.index
        self.home = torch._C._cuda_getCurrentRawStream(self.dev)

    def use(self):
        if torch._C._cuda_getCurrentRawStream(self.dev) != self.home and not torch.cuda.is_current_stream_capturing():
            here = torch.cuda.current_stream(self.dev)
            for t in self.tensors:
                t.record_stream(here)


class _Launcher:
    """The library's entry points on one device's current stream, with the arguments a plan has
    prepared: what a layer's launches cost on the host is then the call itself."""

    def __init__(self, device):
        self.handle = ffi.default_handle(device.index or 0)
        self.dev, self.h, self.lib = self.handle.device, self.handle.ptr, ffi.lib()
        self.stream = 0

    def begin(self):
        """Reads the current stream; returns the context the launches of one pass run in."""
        self.stream = torch._C._cuda_getCurrentRawStream(self.dev)
        return ops._on(torch.device("cuda", self.dev))

    def call(self, fn, *args):
        rc = fn(self.h, self.stream, *args)
        if rc:
            self.handle.check(rc, getattr(fn, "__name__", "kernel call"))


def _product(go, op, a, b, out):
    """out = a b (op 0) or a b^T (op 1), inside go.begin().  In f32 with few output tiles and a long
    contraction the rows kernel has the parts of K that the library's tiles leave to one SM (us, with the
    library's: 32 rows, 768 x 3072 8.9 and 14.6, 1536 x 768 8.5 and 18.2, 512 x 512 5.1 and 8.5; a vocabulary of
    50280 to 768 171 and 165, transposed 156 and 240).  The last size it takes, 96 tiles of 32 x 64, is 64 x 768 x
    3072: 13.9 and 15.8; 96 rows, 144 tiles, are 20.0 and 15.9."""
    M, K = a.shape
    N = out.shape[1]
    if a.dtype == torch.float32 and M >= 12 and K >= 512 and ((M + 31) // 32) * ((N + 63) // 64) <= 96:
        go.call(go.lib.mamba_b200_sgemm_rows, op, a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), None, out.data_ptr(),
                out.stride(0), M, N, K)
    else:
        torch.mm(a, b if op == 0 else b.t(), out=out)


class _Replay:
    """Sequences of a plan's launches that come again with the same addresses, as CUDA graphs.  A model small
    enough for its launches to cost more than its work spends a fifth to a half of a pass between kernels
    (130m, 1021 tokens: 1.96 ms launched one by one, 1.60 replayed; d_model 128, two layers: 0.18 and 0.125;
    a training step of 32 tokens in f32: 7.6 and 6.1 ms).  A sequence is recorded when it comes for the
    third time, if its engine's shelf has room for the `nbytes` of activations that stay with it."""

    def __init__(self, shelf, nbytes):
        self.shelf, self.nbytes, self.seen, self.kept = shelf, nbytes, {}, {}

    def run(self, key, launch):
        """launch() now: by its graph where there is one.  What it returns lives until the next call
        with this key.  launch() reads and writes fixed addresses, apart from what it allocates."""
        shelf, hit = self.shelf, self.kept.get(key)
        shelf.calls += 1
        if hit is not None:
            hit[2].used = shelf.calls
            with ops._on(shelf.device):
                hit[0].replay()
            return hit[1]
        n = self.seen[key] = self.seen.pop(key, 0) + 1
        if len(self.seen) > 64:
            del self.seen[next(iter(self.seen))]
        if n < 3 or not shelf.room(self.nbytes):
            return launch()
        del self.seen[key]
        got = shelf.record(launch)
        if got is None:  # (no memory for it, say: launch() does without, or says so itself)
            return launch()
        self.kept[key] = *got, shelf.put(self, key)
        got[0].replay()
        return got[1]

    def __del__(self):
        for _, _, place in self.kept.values():
            self.shelf.places.discard(place)


class _Shelf:
    """What an engine keeps recorded: no more than KEEP sequences and `limit` bytes of activations, over all
    its plans.  When there is no room, the one whose last use lies PATIENCE calls back gives way; while all
    are in use, further ones are launched one by one, so buffers or lengths in rotation cost at most KEEP
    recordings in PATIENCE calls (a recording takes about as long as five passes)."""

    KEEP, PATIENCE = 16, 1024

    class Place:
        __slots__ = ("replay", "key", "nbytes", "used")

    def __init__(self, device, limit):
        self.device, self.limit, self.places, self.calls, self.stream = device, limit, set(), 0, None

    def room(self, nbytes):
        if nbytes > self.limit:
            return False
        while self.places and (len(self.places) >= self.KEEP or nbytes + sum(p.nbytes for p in self.places) > self.limit):
            last = min(self.places, key=lambda p: p.used)
            if self.calls - last.used < self.PATIENCE:
                return False
            self.places.discard(last)
            owner = last.replay()
            if owner is not None:
                owner.kept.pop(last.key, None)
        return True

    def put(self, replay, key):
        place = self.Place()
        place.replay, place.key, place.nbytes, place.used = weakref.ref(replay), key, replay.nbytes, self.calls
        self.places.add(place)
        return place

    def record(self, launch):
        """(graph, result) of launch(), whose work is still to be done; None where it could not be recorded."""
        if self.stream is None:
            self.stream = _RecordingStream(self.device)
        with torch.cuda.device(self.device):
            graph, here, side = torch.cuda.CUDAGraph(), torch.cuda.current_stream(), self.stream.stream
            side.wait_stream(here)
            try:
                with torch.cuda.stream(side):
                    graph.capture_begin(capture_error_mode="thread_local")
                    try:
                        out = launch()
                    finally:
                        graph.capture_end()
            except RuntimeError:
                return None
            finally:
                here.wait_stream(side)
        return graph, out


class _RecordingStream:
    """A stream that belongs to one engine's recordings.  The workspace that library GEMMs use is one per
    thread and stream, and a recording keeps its address: on a stream of torch's pool, which hands each out
    many times, it could be the workspace of another engine's recording or of a program's own GEMMs, running
    at the same time elsewhere.  An engine's own recordings never run beside each other."""

    spare = {}  # device index -> streams of engines that are gone

    def __init__(self, device):
        self.index = device.index or 0
        free = self.spare.setdefault(self.index, [])
        if free:
            self.raw = free.pop()
        else:
            raw = C.c_void_p()
            with torch.cuda.device(self.index):
                torch.cuda.current_stream().query()  # (the device's context is this thread's own from here on)
                rc = C.CDLL("libcuda.so.1").cuStreamCreate(C.byref(raw), 1)  # CU_STREAM_NON_BLOCKING
            if rc != 0:
                raise RuntimeError(f"cuStreamCreate failed ({rc})")
            self.raw = raw.value
        self.stream = torch.cuda.ExternalStream(self.raw, device=torch.device("cuda", self.index))

    def __del__(self):
        if getattr(self, "raw", None):
            self.spare[self.index].append(self.raw)


class _PrefillPlan:
    """Everything about a prefill of B x T tokens that does not change from call to call: the C
    argument structs of every layer and the weights' views.  Activations come from the caching
    allocator on each call (they are the same for every layer, and are given back); the structs are
    pointed at them again when their addresses have changed."""

    def __init__(self, bb: "GpuMambaBackbone", B: int, T: int):
        w, c = bb.w, bb.cfg
        self.key = _DecodePlan.made_from(bb)
        self.cfg, self.dtype, self.B, self.T, self.where = c, w.dtype, B, T, None  # (not bb: it keeps this plan)
        self.run_on = _Launcher(w.device)
        di, N, dr, xd = c.d_inner, c.d_state, c.dt_rank, c.xdbl_dim
        self.dt, self.es = ops.dtype_code(w.dtype), w.lp.element_size()
        self.ws_bytes = ops.selective_scan_fwd_workspace_bytes(B, T, di, N)
        self.layers = []
        for l in range(c.n_layers):
            p, pm = w.layer(l), w.layer(l, "master")
            cv, sc = ffi.Conv1dArgs(), ffi.SscanFwdArgs()
            cv.dtype, cv.B, cv.T, cv.D, cv.K = self.dt, B, T, di, c.d_conv
            cv.ld_x, cv.ld_u = 2 * di, di
            cv.conv_w, cv.conv_b, cv.conv_state = pm["conv_w"].data_ptr(), pm["conv_b"].data_ptr(), bb.conv[l].data_ptr()
            sc.dtype, sc.B, sc.T, sc.D, sc.N = self.dt, B, T, di, N
            sc.ld_x, sc.ld_delta, sc.delta_softplus, sc.ld_bc, sc.ld_z, sc.z_mode, sc.ld_y = di, di, 1, xd, 2 * di, 1, di
            sc.a_neg, sc.Dp, sc.ssm_state = w.a_neg[l].data_ptr(), pm["d_param"].data_ptr(), bb.ssm[l].data_ptr()
            sc.workspace_bytes = self.ws_bytes
            self.layers.append((pm["norm_w"].data_ptr(), p["in_proj_w"], C.byref(cv), p["x_proj_w"], p["dt_proj_b"],
                                p["dt_proj_w"], C.byref(sc), p["out_proj_w"], cv, sc))
        self.norm_f = w.tail("master")["norm_f"].data_ptr()
        written = B * T * ((c.d_model + 5 * di + xd) * self.es + 4 * c.d_model) + self.ws_bytes
        self.replay, self.ids = _Replay(bb._shelf, written), None
        # (beyond 64 MB of activations the gaps are a few per cent of the work)
        self.launch_bound = w.device.type == "cuda" and written <= 64 << 20

    def point(self, proj, u, xdbl, delta, y, ws):
        di, N, dr, es = self.cfg.d_inner, self.cfg.d_state, self.cfg.dt_rank, self.es
        self.where = (proj, u, xdbl, delta, y, ws)
        for layer in self.layers:
            cv, sc = layer[-2:]
            cv.x, cv.u = proj, u
            sc.x, sc.delta, sc.Bm, sc.Cm = u, delta, xdbl + dr * es, xdbl + (dr + N) * es
            sc.z, sc.y, sc.workspace = proj + di * es, y, ws

    def layers_over(self, temporal, last_only):
        """Every layer over temporal [B, T, d_model] (updated in place); returns the last branch, which
        the final norm adds: rows of every position, or of the last one with its residual rows."""
        c, B, T = self.cfg, self.B, self.T
        dm, di, dr, BT = c.d_model, c.d_inner, c.dt_rank, B * T
        new = lambda *shape: torch.empty(shape, dtype=self.dtype, device=temporal.device)  # noqa: E731
        post, proj, u, xdbl, delta, y = new(BT, dm), new(BT, 2 * di), new(BT, di), new(BT, c.xdbl_dim), new(BT, di), new(BT, di)
        ws = torch.empty(self.ws_bytes, dtype=torch.uint8, device=temporal.device)
        where = (proj.data_ptr(), u.data_ptr(), xdbl.data_ptr(), delta.data_ptr(), y.data_ptr(), ws.data_ptr())
        if where != self.where:
            self.point(*where)
        branch, dtx = post, xdbl[:, :dr]  # the norm reads its branch row before it writes the row over it
        go, lib = self.run_on, self.run_on.lib
        norm, conv, scan = lib.mamba_b200_residual_rmsnorm_fwd, lib.mamba_b200_conv1d_fwd, lib.mamba_b200_sscan_fwd
        res_p, post_p = temporal.data_ptr(), post.data_ptr()
        addmm = torch.addmm
        with go.begin():
            br = None
            for norm_w, w_in, cv, w_x, b_dt, w_dt, sc, w_out, *_ in self.layers:
                go.call(norm, self.dt, res_p, br, norm_w, post_p, None, BT, dm, c.rms_norm_eps)
                _product(go, 0, post, w_in, proj)                           # [BT, 2 di]: x | z in place
                go.call(conv, cv)
                _product(go, 0, u, w_x, xdbl)                               # [BT, dr + 2N]: dt | B | C in place
                addmm(b_dt, dtx, w_dt, out=delta)
                go.call(scan, sc)
                if last_only and w_out is self.layers[-1][7]:
                    break
                _product(go, 0, y, w_out, branch)
                br = post_p
            if last_only:
                return temporal.view(B, T, dm)[:, -1].contiguous(), y.view(B, T, di)[:, -1] @ self.layers[-1][7]
        return temporal, branch

    def final_norm(self, res, branch):
        out = torch.empty(branch.shape, dtype=self.dtype, device=branch.device)
        go = self.run_on
        with go.begin():
            go.call(go.lib.mamba_b200_residual_rmsnorm_fwd, self.dt, res.data_ptr(), branch.data_ptr(), self.norm_f, out.data_ptr(),
                    None, out.shape[0], self.cfg.d_model, self.cfg.rms_norm_eps)
        return out

    def run(self, temporal, last_only=False):
        """The backbone over temporal [B, T, d_model] (updated in place).  last_only: only the last
        position's normalised row is wanted, so the last out_proj and the last norm take that row."""
        if last_only or not self.launch_bound or torch.cuda.is_current_stream_capturing():
            out = self.final_norm(*self.layers_over(temporal, last_only))
            return out if last_only else out.view(self.B, self.T, -1)
        # (the caller keeps the result, so the final norm that writes it is no part of the replay)
        branch = self.replay.run(temporal.data_ptr(), lambda: self.layers_over(temporal, False)[1])
        return self.final_norm(temporal, branch).view(self.B, self.T, -1)


class _DecodePlan:
    """Arguments and workspace of the whole-model decode launch (``mamba_b200_decode_step``) for one
    engine and batch size; ``ok`` is False where the kernel does not take the model or batch."""

    def __init__(self, bb: "GpuMambaBackbone", B: int, lm: "GpuMambaLM | None" = None):
        w, c = bb.w, bb.cfg
        self.key = self.made_from(bb)
        self.handle = ffi.default_handle(w.device.index or 0)
        a = self.args = ffi.DecodeArgs()
        a.dtype = ops.dtype_code(w.dtype)
        a.B, a.batch_capacity, a.d_model, a.d_inner = B, bb.batch, c.d_model, c.d_inner
        a.N, a.K, a.dt_rank, a.n_layers = c.d_state, c.d_conv, c.dt_rank, c.n_layers
        a.vocab, a.eps = (w.vocab if lm else 0), c.rms_norm_eps
        a.lp, a.master, a.a_neg, a.conv_state, a.ssm_state = self.key[:5]
        a.layer_stride = w.layer_size
        offset, o = {}, 0
        for k in _LAYER_FIELDS:
            offset[k], o = o, o + math.prod(w.shapes[k])
        a.o_in_proj, a.o_conv_w, a.o_conv_b = offset["in_proj_w"], offset["conv_w"], offset["conv_b"]
        a.o_x_proj, a.o_dt_proj_w, a.o_dt_proj_b = offset["x_proj_w"], offset["dt_proj_w"], offset["dt_proj_b"]
        a.o_d_param, a.o_out_proj = offset["d_param"], offset["out_proj_w"]
        a.o_norm_f = c.n_layers * w.layer_size
        a.o_embedding = a.o_norm_f + c.d_model
        a.steps = 1
        lib = ffi.lib()
        # the kernel walks the decay rates as one [n_layers, d_inner, N] array
        whole = all(t.data_ptr() == w._a_neg_all[l].data_ptr() for l, t in enumerate(w.a_neg))
        a.workspace_bytes = lib.mamba_b200_decode_workspace_bytes(self.handle.ptr, C.byref(a)) if whole else 0
        self.ok = a.workspace_bytes > 0
        # of the operators' launches where the kernel does not take the model
        self.replay = _Replay(bb._shelf, 4 * B * c.n_layers * (2 * c.d_model + 6 * c.d_inner + c.xdbl_dim))
        if self.ok:
            self.ws = torch.zeros(a.workspace_bytes, dtype=torch.uint8, device=w.device)
            a.workspace = self.ws.data_ptr()
            self.lent = _Lent(self.ws)
            if lm is not None:
                self.res = torch.empty(B, c.d_model, device=w.device)
                a.residual = self.res.data_ptr()
                self.lent = _Lent(self.ws, self.res)
        self._call, self._ref = lib.mamba_b200_decode_step, C.byref(a)

    @staticmethod
    def made_from(bb):
        """All that the structs and recorded launches of a plan hold of their engine: addresses (a layer's
        decay rates may have been replaced by another tensor) and the norm's epsilon."""
        w = bb.w
        return (w.lp.data_ptr(), w.master.data_ptr(), w._a_neg_all.data_ptr(), bb.conv.data_ptr(), bb.ssm.data_ptr(),
                bb.cfg.rms_norm_eps, *[a.data_ptr() for a in w.a_neg])

    def launch(self):
        self.lent.use()
        dev = self.handle.device
        stream = torch.cuda.current_stream(dev).cuda_stream
        if torch.cuda.current_device() == dev:
            rc = self._call(self.handle.ptr, stream, self._ref)
        else:
            with torch.cuda.device(dev):
                rc = self._call(self.handle.ptr, stream, self._ref)
        if rc:
            self.handle.check(rc, "mamba_b200_decode_step")


class GpuMambaBackbone:
    """Prefill + decode over a residual stream [B, T, d_model] f32
    (``GpuMambaBackbone``, src/mamba_ssm/gpu/inference.rs:1515-1855): ``prefill_sequence``
    walks whole sequences, ``step`` one token; both update the recurrent state
    (``conv[L][B,D,K]``, ``ssm[L][B,D,N]`` f32) in place; ``reset`` zeroes it."""

    def __init__(self, weights: MambaWeights, batch: int):
        self.w, self.cfg, self.batch = weights, weights.cfg, batch
        dev, c = weights.device, weights.cfg
        self.conv = torch.zeros(c.n_layers, batch, c.d_inner, c.d_conv, device=dev)
        self.ssm = torch.zeros(c.n_layers, batch, c.d_inner, c.d_state, device=dev)
        self._plans, self._prefills, self._shelf = {}, {}, _Shelf(weights.device, 256 << 20)

    def _plan(self, B):
        """The decode launch for B sequences, rebuilt when a buffer it points at was replaced."""
        p = self._plans.get(B)
        if p is None or p.key != _DecodePlan.made_from(self):
            p = _DecodePlan(self, B)
            if not _capturing(self.w.master):
                if len(self._plans) >= 8:
                    self._plans.clear()
                self._plans[B] = p
        return p

    def reset(self):
        self.conv.zero_()
        self.ssm.zero_()

    def prefill_sequence(self, temporal: torch.Tensor) -> torch.Tensor:
        """temporal [B, T, d_model] f32 (embedded inputs) -> norm_f(residual) [B, T, d_model]
        in the compute dtype.  The input tensor is used as the residual stream (updated in place)."""
        return self._prefill(temporal, False)

    def _prefill(self, temporal, last_only):
        B, T, dm = temporal.shape
        ops._require_cuda(temporal)
        if (temporal.dtype != torch.float32 or not temporal.is_contiguous() or dm != self.cfg.d_model
                or temporal.device != self.w.master.device):
            raise TypeError("temporal is contiguous float32 [B, T, d_model] on the weights' device")
        if B > self.batch:
            raise ValueError(f"{B} sequences, the engine's state holds {self.batch}")
        return self._prefill_plan(B, T).run(temporal, last_only)

    def _prefill_plan(self, B, T):
        p = self._prefills.get((B, T))
        if p is None or p.key != _DecodePlan.made_from(self):
            if len(self._prefills) >= 64:
                self._prefills.clear()
            p = self._prefills[B, T] = _PrefillPlan(self, B, T)
        return p

    def step(self, temporal: torch.Tensor) -> torch.Tensor:
        """One token per sequence: temporal [B, d_model] f32 -> [B, d_model] (compute dtype).  The
        input tensor is used as the residual stream (updated in place).  One launch for the whole
        model where ``mamba_b200_decode_step`` takes it, else the operators one by one."""
        c, w = self.cfg, self.w
        B, dm = temporal.shape
        if dm != c.d_model or temporal.device != w.master.device:
            raise TypeError(f"temporal is [B, {c.d_model}] on {w.master.device}, not {list(temporal.shape)} on {temporal.device}")
        if B > self.batch:
            raise ValueError(f"{B} sequences, the engine's state holds {self.batch}")
        plan = self._plan(B)
        if (plan.ok and temporal.is_cuda and temporal.dtype == torch.float32
                and temporal.is_contiguous() and temporal.data_ptr() % 16 == 0):
            out = torch.empty(B, dm, device=temporal.device, dtype=w.dtype)
            plan.args.residual, plan.args.out = temporal.data_ptr(), out.data_ptr()
            plan.launch()
            return out
        if (temporal.is_cuda and temporal.dtype == torch.float32 and temporal.is_contiguous()
                and not torch.cuda.is_current_stream_capturing()):
            branch = plan.replay.run(temporal.data_ptr(), lambda: self._step_layers(temporal))
        else:
            branch = self._step_layers(temporal)
        return self._step_norm(temporal, branch)  # (the caller keeps it, so it is no part of a replay)

    def _step_operators(self, temporal):
        return self._step_norm(temporal, self._step_layers(temporal))

    def _step_norm(self, temporal, branch):
        return ops.residual_rmsnorm_fwd(temporal, branch, self.w.tail("master")["norm_f"], eps=self.cfg.rms_norm_eps,
                                        out_dtype=self.w.dtype)[0]

    def _step_layers(self, res):
        c, w, B = self.cfg, self.w, res.shape[0]
        di, N, dr = c.d_inner, c.d_state, c.dt_rank
        branch = None
        for l in range(c.n_layers):
            p, pm = w.layer(l), w.layer(l, "master")
            post, _ = ops.residual_rmsnorm_fwd(res, branch, pm["norm_w"], eps=c.rms_norm_eps, out_dtype=w.dtype)
            proj = post @ p["in_proj_w"]
            u = torch.empty(B, di, device=res.device, dtype=w.dtype)
            # x_proj needs u before the scan step can run: conv step first (u_out), then the
            # fused softplus + SSM step + gate on the ready u
            ops.conv1d_fwd(torch.as_strided(proj, (B, 1, di), (2 * di, 2 * di, 1)), pm["conv_w"], pm["conv_b"],
                           self.conv[l], u.view(B, 1, di))
            xdbl = u @ p["x_proj_w"]
            delta = torch.addmm(p["dt_proj_b"], xdbl[:, :dr], p["dt_proj_w"])
            y = ops.selective_scan_step(u, delta, xdbl[:, dr:dr + N], xdbl[:, dr + N:], w.a_neg[l], pm["d_param"],
                                        self.ssm[l], proj[:, di:])
            branch = y @ p["out_proj_w"]
        return branch


class GpuMambaLM:
    """Token-level wrapper with a tied head (``GpuMambaLM``, src/module/gpu_lm.rs:136-679):
    ``prefill`` runs whole prompts through the backbone and returns the logits of the last
    position, ``generate_greedy`` decodes token by token: one launch per token
    (``mamba_b200_decode_step``) where the model allows it.  Otherwise one decode step (embedding
    row, 24-layer step, head GEMM, argmax) is captured in a CUDA graph on first use and replayed,
    as the reference captures its step (src/mamba_ssm/gpu/inference.rs:1608-1630)."""

    def __init__(self, weights: MambaWeights, batch: int):
        if not weights.vocab:
            raise ValueError("the LM needs weights with a vocabulary")
        self.w, self.batch = weights, batch
        self.backbone = GpuMambaBackbone(weights, batch)
        dev = weights.device
        self.next_ids = torch.zeros(batch, dtype=torch.int32, device=dev)
        self.logits = torch.empty(batch, weights.vocab, device=dev, dtype=weights.dtype)
        self._graph = None
        self._dec = None

    def prefill(self, ids: torch.Tensor) -> torch.Tensor:
        """ids [B, T] int32 -> logits of the last position [B, vocab]; leaves the greedy
        next token in ``next_ids``."""
        B, T = ids.shape
        if (B == self.batch and ids.device == self.w.master.device and ids.is_cuda and ids.dtype == torch.int32 and T > 0
                and not torch.cuda.is_current_stream_capturing()):
            p = self.backbone._prefill_plan(B, T)
            if p.launch_bound:
                with torch.cuda.device(ids.device):
                    if p.ids is None:
                        p.ids = torch.empty(B, T, dtype=torch.int32, device=ids.device)
                        p.lent = _Lent(p.ids)
                    p.lent.use()
                    p.ids.copy_(ids)
                    p.replay.run((self.logits.data_ptr(), self.next_ids.data_ptr()), lambda: self._prefill(p.ids))
                return self.logits
        self._prefill(ids.contiguous())
        return self.logits

    def _prefill(self, ids):
        emb = self.w.tail()["embedding"]
        temporal = ops.embedding_gather(emb, ids).view(*ids.shape, -1)
        hidden = self.backbone._prefill(temporal, True)
        torch.matmul(hidden, emb.t(), out=self.logits)
        self.next_ids.copy_(self.logits.argmax(dim=1))

    def _decode_once(self, operators=False):
        emb = self.w.tail()["embedding"]
        temporal = ops.embedding_gather(emb, self.next_ids)
        hidden = self.backbone._step_operators(temporal) if operators else self.backbone.step(temporal)
        torch.matmul(hidden, emb.t(), out=self.logits)
        self.next_ids.copy_(self.logits.argmax(dim=1))

    def generate_greedy(self, n: int, use_graph: bool = True) -> torch.Tensor:
        """n greedy tokens after a prefill; returns them as [B, n] int32.  use_graph=False: operator by
        operator, also where the one-launch kernel would take the step (it needs every SM at once, the
        operators run beside other streams' work)."""
        out = torch.empty(self.batch, n, dtype=torch.int32, device=self.w.device)
        dec = self._dec
        if dec is None or dec.key != _DecodePlan.made_from(self.backbone):
            dec = _DecodePlan(self.backbone, self.batch, self)
            if not _capturing(self.w.master):
                self._dec = dec
        if use_graph and dec.ok and n > 0:
            a = dec.args
            a.next_ids, a.logits, a.steps = self.next_ids.data_ptr(), self.logits.data_ptr(), n
            a.tokens, a.tokens_ld = out.data_ptr(), n
            dec.launch()
            return out
        if use_graph and self._graph is None:
            dev = self.w.device
            keep = (self.backbone.conv.clone(), self.backbone.ssm.clone(), self.next_ids.clone())
            side = torch.cuda.Stream(device=dev)
            side.wait_stream(torch.cuda.current_stream(dev))
            with torch.cuda.stream(side):
                self._decode_once()  # warm-up outside the capture (first-call set-up, cuBLAS workspaces)
            torch.cuda.current_stream(dev).wait_stream(side)
            self._graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self._graph):
                self._decode_once()
            self.backbone.conv.copy_(keep[0])
            self.backbone.ssm.copy_(keep[1])
            self.next_ids.copy_(keep[2])
        for i in range(n):
            out[:, i] = self.next_ids
            if use_graph:
                self._graph.replay()
            else:
                self._decode_once(operators=True)
        return out


class _TrainPlan:
    """What a training step on B x T tokens does not work out again each time: the C argument structs
    of every layer, forward and backward, and the weights' views.  Activations and gradients come from
    the caching allocator in each step; the structs are pointed at them when their addresses changed."""

    class Layer:
        __slots__ = ("norm_w", "g_norm", "w_in", "w_x", "w_x_t", "b_dt", "w_dt", "w_out",
                     "conv", "scan", "conv_b", "scan_b", "structs")

    def __init__(self, w: MambaWeights, B: int, T: int, save: int, shelf: _Shelf):
        c = w.cfg
        self.key, self.B, self.T, self.w = self.made_from(w), B, T, w
        self.run_on = _Launcher(w.device)
        di, N, K, xd, S = c.d_inner, c.d_state, c.d_conv, c.xdbl_dim, save
        self.blocks = (T + S - 1) // S
        self.dt, self.es = ops.dtype_code(w.dtype), w.lp.element_size()
        lib = ffi.lib()
        self.fwd_ws = ops.selective_scan_fwd_workspace_bytes(B, T, di, N)
        self.bwd_ws = max(ops.selective_scan_bwd_workspace_bytes(B, T, di, N),
                          lib.mamba_b200_conv1d_bwd_workspace_bytes(B, T, di, K),
                          lib.mamba_b200_residual_rmsnorm_bwd_workspace_bytes(B * T, c.d_model), 1)
        self.norm_f = w.tail("master")["norm_f"].data_ptr()
        self.fwd_at = self.bwd_at = None
        self.ids = torch.empty(B, T + 1, dtype=torch.int32, device=w.device)
        # few f32 rows: their sum is one more product (of the rows kernel)
        self.ones = torch.ones(B * T, 1, device=w.device) if w.dtype == torch.float32 and B * T <= 32 else None
        self.lent = _Lent(self.ids, *(() if self.ones is None else (self.ones,)))
        a_layer = B * T * (4 * (c.d_model + 1) + self.es * (c.d_model + 5 * di + xd)) + 4 * B * self.blocks * di * N
        written = c.n_layers * a_layer + B * T * self.es * (w.vocab or 0) + self.fwd_ws + self.bwd_ws
        # (beyond 512 MB of activations the gaps are a few per cent of the work)
        self.launch_bound = w.device.type == "cuda" and written <= 512 << 20
        self.replay = _Replay(shelf, written)
        self.layers = []
        for l in range(c.n_layers):
            p, pm, g, lay = w.layer(l), w.layer(l, "master"), w.layer(l, "grad"), self.Layer()
            lay.norm_w, lay.g_norm = pm["norm_w"].data_ptr(), g["norm_w"].data_ptr()
            lay.w_in, lay.w_x, lay.b_dt, lay.w_dt, lay.w_out = (p[k] for k in ("in_proj_w", "x_proj_w", "dt_proj_b", "dt_proj_w", "out_proj_w"))
            lay.w_x_t = lay.w_x.t()
            cv, sc, cb, sb = ffi.Conv1dArgs(), ffi.SscanFwdArgs(), ffi.Conv1dArgs(), ffi.SscanBwdArgs()
            for q in (cv, cb):
                q.dtype, q.B, q.T, q.D, q.K, q.ld_x = self.dt, B, T, di, K, 2 * di
                q.conv_w, q.conv_b = pm["conv_w"].data_ptr(), pm["conv_b"].data_ptr()
            cv.ld_u = cb.ld_du = di
            cb.ld_dx, cb.dconv_w, cb.dconv_b, cb.workspace_bytes = 2 * di, g["conv_w"].data_ptr(), g["conv_b"].data_ptr(), self.bwd_ws
            for q in (sc, sb):
                q.dtype, q.B, q.T, q.D, q.N = self.dt, B, T, di, N
                q.ld_delta, q.delta_softplus, q.ld_bc, q.ld_z, q.z_mode = di, 1, xd, 2 * di, 1
                q.a_neg, q.Dp, q.save_stride = w.a_neg[l].data_ptr(), pm["d_param"].data_ptr(), S
            sc.ld_x = sc.ld_y = sb.ld_u = sb.ld_dy = sb.ld_du = sb.ld_ddelta = di
            sc.workspace_bytes, sb.workspace_bytes, sb.ld_dz = self.fwd_ws, self.bwd_ws, 2 * di
            sb.dA_log, sb.dD = g["a_log"].data_ptr(), g["d_param"].data_ptr()
            lay.structs = (cv, sc, cb, sb)
            lay.conv, lay.scan, lay.conv_b, lay.scan_b = (C.byref(q) for q in lay.structs)
            self.layers.append(lay)

    @staticmethod
    def made_from(w):
        return (w.lp.data_ptr(), w.master.data_ptr(), w.grad.data_ptr(), w.cfg.rms_norm_eps, *[a.data_ptr() for a in w.a_neg])

    def _at(self, l, proj, u, xdbl, delta, cs):
        """Addresses of layer l's saved x, z, u, B, C, delta and block states."""
        c, es, BT = self.w.cfg, self.es, self.B * self.T
        di, N, xd = c.d_inner, c.d_state, c.xdbl_dim
        x, b = proj + es * BT * 2 * di * l, xdbl + es * (BT * xd * l + c.dt_rank)
        return (x, x + es * di, u + es * BT * di * l, b, b + es * N, delta + es * BT * di * l,
                cs + 4 * self.B * self.blocks * di * N * l)

    def point_forward(self, proj, u, xdbl, delta, y, cs, ws):
        at = tuple(t.data_ptr() for t in (proj, u, xdbl, delta, y, cs, ws))
        if at == self.fwd_at:
            return
        self.fwd_at = at
        step = self.es * self.B * self.T * self.w.cfg.d_inner
        for l, lay in enumerate(self.layers):
            cv, sc = lay.structs[:2]
            x, z, u_l, b, c_, d, s_ = self._at(l, at[0], at[1], at[2], at[3], at[5])
            cv.x, cv.u = x, u_l
            sc.x, sc.delta, sc.Bm, sc.Cm, sc.z, sc.y, sc.chunk_states, sc.workspace = u_l, d, b, c_, z, at[4] + step * l, s_, at[6]

    def point_backward(self, acts, d_y, d_u, d_delta, d_proj, d_bc, ws):
        at = tuple(t.data_ptr() for t in (acts["proj"], acts["u"], acts["xdbl"], acts["delta"], acts["cs"], d_y, d_u, d_delta, d_proj, d_bc, ws))
        if at == self.bwd_at:
            return
        self.bwd_at = at
        dz = at[8] + self.es * self.w.cfg.d_inner
        dc = at[9] + 4 * self.B * self.T * self.w.cfg.d_state
        for l, lay in enumerate(self.layers):
            cb, sb = lay.structs[2:]
            x, z, u_l, b, c_, d, s_ = self._at(l, *at[:5])
            sb.u, sb.delta, sb.Bm, sb.Cm, sb.z, sb.chunk_states, sb.dy = u_l, d, b, c_, z, s_, at[5]
            sb.d_u, sb.d_delta, sb.d_z, sb.dBm, sb.dCm, sb.workspace = at[6], at[7], dz, at[9], dc, at[10]
            cb.x, cb.d_u, cb.d_x, cb.workspace = x, at[6], at[8], at[10]


class MambaLMTrainer:
    """A next-token training step on the device: embedding gather, the backbone forward
    with block-boundary state saves, tied-head logits, softmax cross-entropy, the manual
    backward (scan / conv / norm backward kernels of this library, GEMM gradients through
    cuBLAS), a bucketed gradient all-reduce that overlaps the rest of the backward, and
    fused AdamW.  ``forward`` / ``backward_step`` / ``step`` follow ``MambaTrainer``
    (src/mamba_ssm/gpu/trainer.rs:437-481); ``accumulate_only`` is its
    ``BackwardOpts::accumulate_only`` (trainer.rs:176-206) for micro-batching."""

    SAVE = 32  # steps between saved scan states

    def __init__(self, weights: MambaWeights, lr=3e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, group=None):
        if not weights.vocab:
            raise ValueError("the LM trainer needs weights with a vocabulary")
        self.w, self.cfg, self.group = weights, weights.cfg, group
        self.lr, self.betas, self.eps, self.wd = lr, betas, eps, weight_decay
        self.m = torch.zeros_like(weights.master)
        self.v = torch.zeros_like(weights.master)
        self.t = 0
        self.bias = torch.ones(2, device=weights.device)
        self._acts = None
        self._pending = 0
        self._plans, self._shelf = {}, _Shelf(weights.device, 1 << 30)

    # ---- forward ----
    def forward(self, ids: torch.Tensor) -> torch.Tensor:
        """ids [B, T+1] int32: predicts token t+1 from tokens <= t.  Returns the mean loss
        (a device scalar) and keeps what the backward needs."""
        c, w = self.cfg, self.w
        B, T1 = ids.shape
        T = T1 - 1
        dm, BT, L = c.d_model, B * T, c.n_layers
        dev, plan = w.device, self._plan(B, T)
        emb = w.tail()["embedding"]
        inp = ids[:, :-1].contiguous()
        go, lib = plan.run_on, plan.run_on.lib
        new = lambda *shape: torch.empty(shape, dtype=w.dtype, device=dev)  # noqa: E731
        f32 = lambda *shape: torch.empty(shape, device=dev)  # noqa: E731
        # saved activations, one tensor per kind over all layers: residual stream as each norm saw it
        # ([0] is the embedding), row rms, normalised rows, x | z, u, dt | B | C, delta, y, block states
        di = c.d_inner
        res, rms = f32(L + 1, BT, dm), f32(L + 1, BT)
        post, proj, u, xdbl = new(L, BT, dm), new(L, BT, 2 * di), new(L, BT, di), new(L, BT, c.xdbl_dim)
        delta, y, cs = new(L, BT, di), new(L, BT, di), f32(L, B, plan.blocks, di, c.d_state)
        branch, hidden, ws = new(BT, dm), new(BT, dm), torch.empty(plan.fwd_ws, dtype=torch.uint8, device=dev)
        plan.point_forward(proj, u, xdbl, delta, y, cs, ws)
        norm, conv, scan = lib.mamba_b200_residual_rmsnorm_fwd_to, lib.mamba_b200_conv1d_fwd, lib.mamba_b200_sscan_fwd
        ops.embedding_gather(emb, inp, res[0])
        addmm, dr = torch.addmm, c.dt_rank
        res_p, rms_p, post_p, branch_p = res.data_ptr(), rms.data_ptr(), post.data_ptr(), branch.data_ptr()
        with go.begin():
            acts = list(zip(post.unbind(), proj.unbind(), u.unbind(), xdbl.unbind(), delta.unbind(), y.unbind()))
            for l, (lay, (post_l, proj_l, u_l, xdbl_l, delta_l, y_l)) in enumerate(zip(plan.layers, acts)):
                # the stream this layer's norm saw is kept in res[l]; the embedding is there already
                go.call(norm, plan.dt, res_p + 4 * BT * dm * max(l - 1, 0), branch_p if l else None, lay.norm_w,
                        res_p + 4 * BT * dm * l, post_p + plan.es * BT * dm * l, rms_p + 4 * BT * l, BT, dm, c.rms_norm_eps)
                _product(go, 0, post_l, lay.w_in, proj_l)
                go.call(conv, lay.conv)
                _product(go, 0, u_l, lay.w_x, xdbl_l)
                addmm(lay.b_dt, xdbl_l[:, :dr], lay.w_dt, out=delta_l)
                go.call(scan, lay.scan)
                _product(go, 0, y_l, lay.w_out, branch)
            go.call(norm, plan.dt, res_p + 4 * BT * dm * (L - 1), branch_p, plan.norm_f, res_p + 4 * BT * dm * L,
                    hidden.data_ptr(), rms_p + 4 * BT * L, BT, dm, c.rms_norm_eps)
        logits = hidden @ emb.t()                                  # tied head, [BT, V]
        tgt = ids[:, 1:].contiguous().view(-1)
        # the gradient takes the logits' place: every row is read before it is written
        loss_rows, dlogits = ops.softmax_xent(logits, tgt, grad_scale=1.0 / BT, dlogits=logits)
        self._acts = dict(layers=acts, res=res, rms=rms, proj=proj, u=u, xdbl=xdbl, delta=delta, cs=cs, hidden=hidden,
                          dlogits=dlogits, inp=inp, B=B, T=T, plan=plan)
        return loss_rows.sum() / BT

    def _plan(self, B, T):
        p = self._plans.get((B, T))
        if p is None or p.key != _TrainPlan.made_from(self.w):
            p = _TrainPlan(self.w, B, T, self.SAVE, self._shelf)
            if not _capturing(self.w.master):
                if len(self._plans) >= 16:
                    self._plans.clear()
                self._plans[B, T] = p
        return p

    def _accumulate(self, g, a, b):
        """g (f32) += a.T @ b, the product accumulated into g by the GEMM itself."""
        # up to 32 rows are one pass over the tiles of the rows kernel (us, with the library's: 32 rows, 768 x 3072 6.2
        # and 8.9, 1536 x 80 2.9 and 4.0, 50280 x 768 82 and 101); 33 are two (10.0 and
        # 9.9, 4.2 and 4.3, 131 and 105)
        if a.dtype == torch.float32 and a.shape[0] <= 32:
            go = self._acts["plan"].run_on
            with go.begin():
                go.call(go.lib.mamba_b200_sgemm_rows, 2, a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), None,
                        g.data_ptr(), g.stride(0), g.shape[0], g.shape[1], a.shape[0])
        elif a.dtype == torch.float32:
            g.addmm_(a.t(), b)
        else:
            torch.addmm(g, a.t(), b, out_dtype=torch.float32, out=g)

    # ---- backward + optimiser ----
    def backward_step(self, accumulate_only: bool = False):
        self._gradients(accumulate_only)
        if not accumulate_only:
            self._update()

    def _gradients(self, accumulate_only):
        c, w, a = self.cfg, self.w, self._acts
        if a is None:
            raise RuntimeError("backward_step needs a forward first")
        B, T, plan = a["B"], a["T"], a["plan"]
        di, N, dr, dm, L, BT = c.d_inner, c.d_state, c.dt_rank, c.d_model, c.n_layers, B * T
        dev, dt = w.device, w.dtype
        red = None if accumulate_only else BucketedGradReducer(w.grad, w.bucket_bounds(), group=self.group, average=True)
        emb = w.tail()["embedding"]
        gt = w.tail("grad")
        dl, acc = a["dlogits"], self._accumulate
        acc(gt["embedding"], dl, a["hidden"])                       # head weight gradient
        d_post = torch.empty(BT, dm, dtype=dt, device=dev)          # here of the final norm
        with plan.run_on.begin():
            _product(plan.run_on, 0, dl, emb, d_post)
        a["dlogits"] = dl = None
        new = lambda *shape: torch.empty(shape, dtype=dt, device=dev)  # noqa: E731
        d_res = torch.zeros(BT, dm, device=dev)
        d_y, d_u, d_delta, d_proj, d_xdbl = new(BT, di), new(BT, di), new(BT, di), new(BT, 2 * di), new(BT, c.xdbl_dim)
        d_bc = torch.empty(2, BT, N, device=dev)
        d_out = d_res if dt == torch.float32 else new(BT, dm)
        ws = torch.empty(plan.bwd_ws, dtype=torch.uint8, device=dev)
        plan.point_backward(a, d_y, d_u, d_delta, d_proj, d_bc, ws)
        go, lib = plan.run_on, plan.run_on.lib
        norm, conv, scan = lib.mamba_b200_residual_rmsnorm_bwd, lib.mamba_b200_conv1d_bwd, lib.mamba_b200_sscan_bwd
        res_p, rms_p, dres_p, ws_p = a["res"].data_ptr(), a["rms"].data_ptr(), d_res.data_ptr(), ws.data_ptr()
        d_dt_in, d_bc_out, d_bc_in = d_xdbl[:, :dr], d_xdbl[:, dr:].view(BT, 2, N), d_bc.transpose(0, 1)
        addmm = torch.addmm
        with go.begin():
            dp = d_post.data_ptr()
            go.call(norm, plan.dt, dp, res_p + 4 * BT * dm * L, plan.norm_f, rms_p + 4 * BT * L, dres_p, gt["norm_f"].data_ptr(),
                    BT, dm, ws_p, plan.bwd_ws)
            for l in range(L - 1, -1, -1):
                lay, g = plan.layers[l], w.layer(l, "grad")
                post, proj, u, xdbl, delta, y = a["layers"][l]
                if d_out is not d_res:
                    d_out.copy_(d_res)                              # gradient of this layer's branch output
                acc(g["out_proj_w"], y, d_out)
                _product(go, 1, d_out, lay.w_out, d_y)
                go.call(scan, lay.scan_b)
                if plan.ones is not None:
                    plan.lent.use()
                    acc(g["dt_proj_b"].view(1, di), plan.ones, d_delta)
                else:
                    g["dt_proj_b"].add_(torch.sum(d_delta, 0, dtype=torch.float32))
                acc(g["dt_proj_w"], xdbl[:, :dr], d_delta)
                _product(go, 1, d_delta, lay.w_dt, d_dt_in)
                d_bc_out.copy_(d_bc_in)
                acc(g["x_proj_w"], u, d_xdbl)
                addmm(d_u, d_xdbl, lay.w_x_t, out=d_u)              # backward_mixed.rs:350-580
                go.call(conv, lay.conv_b)
                acc(g["in_proj_w"], post, d_proj)
                _product(go, 1, d_proj, lay.w_in, d_post)
                go.call(norm, plan.dt, dp, res_p + 4 * BT * dm * l, lay.norm_w, rms_p + 4 * BT * l, dres_p, lay.g_norm,
                        BT, dm, ws_p, plan.bwd_ws)
                if red is not None:
                    red.bucket_ready(l)                              # its all-reduce runs under layers l-1 .. 0
        # embedding rows: the residual gradient flows into the gathered rows
        gt["embedding"].index_add_(0, a["inp"].view(-1), d_res)
        self._acts = None
        self._pending += 1
        if red is not None:
            red.bucket_ready(L)
            red.finish()

    def _update(self):
        """AdamW on the gradients in the arena, which is zero again afterwards."""
        w = self.w
        if self._pending > 1:
            w.grad.div_(self._pending)
        self._pending = 0
        self.t += 1
        b1, b2 = self.betas
        self.bias[:1].fill_(1.0 / (1.0 - b1 ** self.t))
        self.bias[1:].fill_(1.0 / (1.0 - b2 ** self.t))
        ops.adamw_step(w.master, w.grad, self.m, self.v, self.bias, lr=self.lr, beta1=b1, beta2=b2, eps=self.eps,
                       weight_decay=self.wd, param_lp=None if w.lp is w.master else w.lp)
        w.refresh_a_neg()
        w.grad.zero_()

    def _loss_and_gradients(self, ids):
        loss = self.forward(ids)
        self._gradients(False)
        return loss

    def step(self, ids: torch.Tensor) -> torch.Tensor:
        B, T1 = ids.shape
        if (ids.device == self.w.master.device and ids.is_cuda and ids.dtype == torch.int32 and B > 0 and T1 > 1
                and self._pending == 0 and self._acts is None
                and not torch.distributed.is_initialized() and not torch.cuda.is_current_stream_capturing()):
            plan = self._plan(B, T1 - 1)
            if plan.launch_bound:
                with torch.cuda.device(self.w.device):
                    plan.lent.use()
                    plan.ids.copy_(ids)
                    # (the update stays outside: a schedule changes its numbers from step to step)
                    loss = plan.replay.run((), lambda: self._loss_and_gradients(plan.ids)).clone()
                    self._update()
                    return loss
        loss = self.forward(ids)
        self.backward_step()
        return loss
