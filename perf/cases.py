"""The work a user of this framework gives it: decoding, prefill, training and the scans themselves.

Each case is a dict of plain values; `prepare` makes what a program holds before the call (weights,
engines, inputs, lent workspaces), `run` is one call through the public entry points.  Seven kinds:

  step       GpuMambaBackbone.step: one token per sequence, layer by layer (control loops, small models)
  decode     GpuMambaLM.generate_greedy: n tokens per sequence after a prompt
  prefill    GpuMambaLM.prefill (token ids) or GpuMambaBackbone.prefill_sequence (ready input rows)
  train      MambaLMTrainer.step: forward, cross-entropy, backward, AdamW
  scan_fwd   selective_scan_fwd with gate and carried state
  scan_bwd   selective_scan_bwd from saved block states
  m3_fwd / m3_bwd / m3_window
             m3_ssd_fwd over whole sequences, m3_ssd_bwd, and m3_ssd_fwd continuing a carried state
"""
import math

import torch

import mamba_rs_b200 as mb

_DT = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
_SIZE = {"bf16": 2, "f16": 2, "f32": 4}
N, KCONV, STRIDE = 16, 4, 32  # d_state and d_conv of every Mamba-1 configuration here; steps between saved states
_LM_130M = dict(d_model=768, layers=24, vocab=50280)


def listed():
    return [
        # the smallest call: one step of the default 3-layer model for one sequence, f32
        dict(name="step_d128_b1_f32", kind="step", d_model=128, layers=3, B=1, dtype="f32"),
        # serving: greedy decoding of 8 sequences at the 130m architecture
        dict(name="decode_130m_b8", kind="decode", B=8, n=16, dtype="bf16", **_LM_130M),
        # the small f32 backbone over a batch of input rows
        dict(name="prefill_d128_b4_t512_f32", kind="prefill", d_model=128, layers=2, vocab=0, B=4, T=512, dtype="f32"),
        # one prompt of a ragged length, 130m architecture: time to the first token
        dict(name="prefill_130m_b1_t1021", kind="prefill", B=1, T=1021, dtype="bf16", **_LM_130M),
        # a full batch of prompts
        dict(name="prefill_130m_b8_t2048", kind="prefill", B=8, T=2048, dtype="bf16", **_LM_130M),
        # fine-tuning on one short sequence in f32: a training step made of small launches
        dict(name="train_130m_b1_t32_f32", kind="train", B=1, T=32, dtype="f32", **_LM_130M),
        # pre-training shard: the 2.8b layer shape, 4 of its layers, two sequences of 8192
        dict(name="train_2p8b_l4_b2_t8192", kind="train", d_model=2560, layers=4, vocab=50280, B=2, T=8192, dtype="bf16"),
        # the standalone scan, trained (general) decay rates, forward and backward
        dict(name="scan_fwd_b16_t2048_d1536", kind="scan_fwd", B=16, T=2048, D=1536, a="trained", dtype="bf16"),
        dict(name="scan_bwd_b16_t2048_d1536", kind="scan_bwd", B=16, T=2048, D=1536, a="trained", dtype="bf16"),
        # one Mamba-3 layer over long sequences, forward and backward
        dict(name="m3_fwd_b8_t4096_h32", kind="m3_fwd", B=8, T=4096, nh=32, hd=64, N=128, dtype="bf16"),
        dict(name="m3_bwd_b8_t4096_h32", kind="m3_bwd", B=8, T=4096, nh=32, hd=64, N=128, dtype="bf16"),
        # one Mamba-3 layer taking the next window of a stream: the state of the last call carries on
        dict(name="m3_window_b8_t256_h32", kind="m3_window", B=8, T=256, nh=32, hd=64, N=128, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _model(rng, kind):
    """A model's sizes: width a multiple of 8, depth as deep as that width is used with."""
    d = 8 * _log(rng, 8, 128)
    c = dict(kind=kind, d_model=d, layers=_log(rng, 2, 24), dtype=rng.choice(("bf16", "bf16", "f16", "f32")))
    if kind in ("decode", "train") or (kind == "prefill" and rng.random() < 0.7):
        c["vocab"] = _log(rng, 500, 50280)
    elif kind == "prefill":
        c["vocab"] = 0
    return c


def draw(rng):
    """One more case of the kinds above; sizes that would cost more than the largest listed case are drawn again."""
    kind = rng.choice(("step", "decode", "prefill", "train", "scan_fwd", "scan_bwd", "m3_fwd", "m3_bwd", "m3_window"))
    for _ in range(1000):
        if kind in ("step", "decode", "prefill", "train"):
            c = _model(rng, kind)
            if kind == "step":
                c.update(B=_log(rng, 1, 64))
            elif kind == "decode":
                c.update(B=_log(rng, 1, 32), n=rng.randint(4, 24))
            else:
                c.update(B=_log(rng, 1, 16), T=_log(rng, 16, 4096))
                if kind == "train":  # no loss scaler: bf16 for the larger steps, f32 for short and deep ones
                    c["dtype"] = "bf16" if c["B"] * c["T"] >= 512 and c["layers"] <= 6 else "f32"
                flops = work(c)["flops"] * (1 if c["dtype"] != "f32" else 12)
                if not 1e9 < flops < 8e12 or c["B"] * c["T"] * c.get("vocab", 0) > 1.2e9:
                    continue
            return c
        if kind.startswith("scan"):
            D = 8 * _log(rng, 8, 640) if rng.random() < 0.8 else _log(rng, 64, 5120) | 1
            c = dict(kind=kind, B=_log(rng, 1, 16), T=_log(rng, 64, 8192), D=D, a=rng.choice(("trained", "trained", "init")),
                     dtype=rng.choice(("bf16", "bf16", "f16", "f32")))
            if 5e5 < c["B"] * c["T"] * D < 5.2e7:
                return c
        else:
            c = dict(kind=kind, B=_log(rng, 1, 8), T=_log(rng, 1 if kind == "m3_window" else 64, 1024 if kind == "m3_window" else 8192),
                     nh=_log(rng, 2, 32), hd=rng.choice((32, 64, 64)), N=rng.choice((64, 128, 128)), dtype=rng.choice(("bf16", "bf16", "f16")))
            if 64 <= c["B"] * c["T"] * c["nh"] <= 1.05e6:
                return c
    raise RuntimeError("no case in range")


# ---------------------------------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------------------------------

def _weights(c, dev, seed, trained):
    cfg = mb.MambaConfig(d_model=c["d_model"], n_layers=c["layers"], d_state=N, d_conv=KCONV)
    w = mb.MambaWeights(cfg, dev, dtype=_DT[c["dtype"]], vocab=c.get("vocab") or None).init_random(seed)
    if trained:
        # after training the decay rates have left the exact -1..-16 of the initialisation, and the
        # tied head tells tokens apart by more than the last bit of a 16-bit logit
        g = torch.Generator(device=dev).manual_seed(seed + 1)
        for l in range(c["layers"]):
            a = w.layer(l, "master")["a_log"]
            a.add_(0.1 * torch.randn(a.shape, device=dev, generator=g))
        if w.vocab:
            w.tail("master")["embedding"].mul_(50.0)
        w.refresh()
    return w


def prepare(case, seed):
    c, kind = case, case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    dt = _DT[c["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device=dev, generator=g)  # noqa: E731
    ids = lambda *s: torch.randint(0, c["vocab"], s, device=dev, dtype=torch.int32, generator=g)  # noqa: E731
    s = dict(kind=kind)
    if kind == "step":
        w = _weights(c, dev, seed, trained=True)
        bb = mb.GpuMambaBackbone(w, c["B"])
        s.update(bb=bb, x=rn(c["B"], c["d_model"]))
        bb.prefill_sequence(rn(c["B"], 32, c["d_model"]))  # some history in the recurrent state
    elif kind == "decode":
        lm = mb.GpuMambaLM(_weights(c, dev, seed, trained=True), c["B"])
        lm.prefill(ids(c["B"], 32))
        lm.generate_greedy(1)  # a server's first token
        s.update(lm=lm, n=c["n"])
    elif kind == "prefill":
        w = _weights(c, dev, seed, trained=True)
        if c["vocab"]:
            s.update(lm=mb.GpuMambaLM(w, c["B"]), ids=ids(c["B"], c["T"]))
        else:
            s.update(bb=mb.GpuMambaBackbone(w, c["B"]), x=rn(c["B"], c["T"], c["d_model"]))
    elif kind == "train":
        s.update(tr=mb.MambaLMTrainer(_weights(c, dev, seed, trained=False), lr=1e-5), ids=ids(c["B"], c["T"] + 1))
    elif kind in ("scan_fwd", "scan_bwd"):
        B, T, D = c["B"], c["T"], c["D"]
        bias = torch.exp(torch.rand(D, device=dev, generator=g) * math.log(100.0) + math.log(1e-3))
        bias = bias + torch.log(-torch.expm1(-bias))  # inverse softplus of a log-uniform step in [1e-3, 1e-1]
        delta = rn(B, T, D).mul_(0.5).add_(bias).to(dt)
        if c["a"] == "trained":
            a = -torch.exp(torch.rand(D, N, device=dev, generator=g) * math.log(32.0) + math.log(0.5))
        else:
            a = -torch.arange(1.0, N + 1, device=dev).repeat(D, 1)
        args = [rn(B, T, D).to(dt), delta, rn(B, T, N).to(dt), rn(B, T, N).to(dt), a.contiguous(), torch.ones(D, device=dev)]
        s.update(args=args, z=rn(B, T, D).to(dt))
        if kind == "scan_fwd":
            s.update(h=rn(B, D, N), ws=torch.empty(max(mb.selective_scan_fwd_workspace_bytes(B, T, D, N), 1), dtype=torch.uint8, device=dev))
        else:
            cs = torch.empty(B, (T + STRIDE - 1) // STRIDE, D, N, device=dev)
            mb.selective_scan_fwd(*args, s["z"], chunk_states=cs, save_stride=STRIDE)
            s.update(dy=rn(B, T, D).to(dt), cs=cs,
                     ws=torch.empty(mb.selective_scan_bwd_workspace_bytes(B, T, D, N), dtype=torch.uint8, device=dev))
    else:
        B, T, nh, hd, n = c["B"], c["T"], c["nh"], c["hd"], c["N"]
        u = lambda *sh: torch.rand(*sh, device=dev, generator=g)  # noqa: E731
        bias = torch.exp(u(nh) * math.log(100.0) + math.log(1e-3))
        bias = bias + torch.log(-torch.expm1(-bias))
        step = torch.nn.functional.softplus(0.5 * rn(B, T, nh) + bias)
        rate = -torch.exp(u(nh) * math.log(16.0))
        sc = n ** -0.25
        s["args"] = [rn(B, T, nh * hd).to(dt), (sc * rn(B, T, nh, n)).to(dt), (sc * rn(B, T, nh, n)).to(dt), step.contiguous(),
                     torch.sigmoid(rn(B, T, nh)), (rate * step).contiguous(), torch.ones(nh, device=dev)]
        if kind == "m3_bwd":
            need = mb.ffi.lib().mamba_b200_m3_ssd_bwd_workspace_bytes_for(mb.dtype_code(dt), B, T, nh, hd, n)
            s.update(dy=rn(B, T, nh * hd).to(dt), ws=torch.empty(max(need, 256), dtype=torch.uint8, device=dev))
        else:
            s["state"] = dict(ssm_state=rn(B, nh, hd, n), k_state=sc * rn(B, nh, n), v_state=rn(B, nh, hd))
    return s


# ---------------------------------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "step":
        bb = s["bb"]
        out = bb.step(s["x"].clone())  # the engine takes its input rows as the residual stream
        return dict(out=out, conv=bb.conv, ssm=bb.ssm)
    if kind == "decode":
        lm = s["lm"]
        tokens = lm.generate_greedy(s["n"])
        return dict(tokens=tokens, logits=lm.logits, conv=lm.backbone.conv, ssm=lm.backbone.ssm)
    if kind == "prefill":
        if "lm" in s:
            lm = s["lm"]
            lm.backbone.reset()
            return dict(logits=lm.prefill(s["ids"]), next_ids=lm.next_ids, conv=lm.backbone.conv, ssm=lm.backbone.ssm)
        bb = s["bb"]
        bb.reset()
        out = bb.prefill_sequence(s["x"].clone())
        return dict(out=out, conv=bb.conv, ssm=bb.ssm)
    if kind == "train":
        tr = s["tr"]
        loss = tr.step(s["ids"])
        return dict(loss=loss, master=tr.w.master, compute=tr.w.lp, m=tr.m, v=tr.v)
    if kind == "scan_fwd":
        y = mb.selective_scan_fwd(*s["args"], s["z"], ssm_state=s["h"], workspace=s["ws"])
        return dict(y=y, h=s["h"])
    if kind == "scan_bwd":
        return mb.selective_scan_bwd(*s["args"], s["dy"], s["cs"], STRIDE, s["z"], workspace=s["ws"])
    if kind == "m3_bwd":
        return mb.m3_ssd_bwd(*s["args"], s["dy"], workspace=s["ws"])
    y = mb.m3_ssd_fwd(*s["args"], carry_in=kind == "m3_window", **s["state"])
    return dict(y=y, **s["state"])


# ---------------------------------------------------------------------------------------------------
# what a call cannot do without, and how far two right answers may lie apart
# ---------------------------------------------------------------------------------------------------

def _layer_sizes(c):
    d = c["d_model"]
    di, dr = 2 * d, (d + 15) // 16
    gemm = d * 2 * di + di * (dr + 2 * N) + dr * di + di * d      # weights that meet every token
    rest = d + di * (KCONV + 1) + di + di * N + di                # norm, conv, dt bias, a_log, D
    return di, gemm, rest


def work(case):
    c, kind, e = case, case["kind"], _SIZE[case["dtype"]]
    if kind in ("step", "decode", "prefill", "train"):
        di, gemm, rest = _layer_sizes(c)
        L, d, V, B = c["layers"], c["d_model"], c.get("vocab", 0), c["B"]
        weights = e * (L * gemm + V * d) + 4 * L * rest
        state = 2 * 4 * L * B * di * (N + KCONV)
        if kind in ("step", "decode"):
            n = c.get("n", 1)
            rows = B * d * (4 + e) + B * V * e
            return {"bytes": n * (weights + state + rows), "flops": n * B * (2 * (L * gemm + V * d) + L * di * N * 6)}
        T = c["T"]
        if kind == "prefill":
            return {"bytes": weights + state / 2 + B * T * 4 + (0 if V else B * T * d * (4 + e)) + B * V * e,
                    "flops": B * T * L * (2 * gemm + di * (6 * N + 2 * KCONV)) + 2 * B * V * d}
        params = L * (gemm + rest) + d + V * d
        # weights, AdamW's three arenas read and written, the compute copy written, and each layer's
        # saved activations (normalised input, x | z, u, dt | B | C, delta, y) written once and read once
        acts = B * T * (L * e * (d + 2 * di + di + (d + 15) // 16 + 2 * N + di + di) + 2 * e * V)
        return {"bytes": params * (4 * 6 + e) + 2 * acts, "flops": 3 * B * T * (L * (2 * gemm + di * 6 * N) + 2 * V * d)}
    if kind in ("scan_fwd", "scan_bwd"):
        B, T, D = c["B"], c["T"], c["D"]
        if kind == "scan_fwd":
            return {"bytes": 4 * e * B * T * D + 2 * e * B * T * N + 4 * D * (N + 1) + 8 * B * D * N, "flops": B * T * D * (6 * N + 12)}
        blocks = (T + STRIDE - 1) // STRIDE
        return {"bytes": 7 * e * B * T * D + (2 * e + 8) * B * T * N + 4 * B * blocks * D * N, "flops": B * T * D * (18 * N + 30)}
    B, T, nh, hd, n = c["B"], c["T"], c["nh"], c["hd"], c["N"]
    x, kq, v = B * T * nh * hd, B * T * nh * n, B * T * nh
    state = 4 * B * nh * (hd * n + n + hd)
    if kind == "m3_bwd":
        return {"bytes": 3 * e * x + 2 * e * kq + 8 * kq + 24 * v, "flops": 2.0 * B * T * nh * (9 * hd * n)}
    return {"bytes": 2 * e * x + 2 * e * kq + 12 * v + (2 if kind == "m3_window" else 1) * state, "flops": 2.0 * B * T * nh * (3 * hd * n)}


def tolerance(case):
    """16-bit storage rounds every activation to 8 (bf16) or 11 (f16) bits, and each layer of a model adds
    its own roundings; f32 storage leaves the order of the sums and the exponentials' last bits."""
    if case["dtype"] == "f32":
        return {"rel": 1e-4 if "layers" in case else 2e-5, "max": 5e-2 if case["kind"] == "train" else 1e-2}
    if case["kind"] == "train":  # gradients of one layer carry the roundings of all the others, the moments their squares
        return {"rel": 3e-2, "max": 0.95}
    if "layers" in case:
        return {"rel": 2e-2, "max": 0.8}
    return {"rel": 1e-2, "max": 0.4}
