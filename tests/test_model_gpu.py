"""The host-side engines (mamba_rs_b200.model) against the CPU oracle's backbone prefill
(d_model 128, 2 layers, f32: every layer's GEMMs, conv, scan, gate, norm chained) and
against a float64 torch restatement with autograd for the training step's gradients."""
import numpy as np
import pytest

import oracle
from helpers import rel_err

pytestmark = pytest.mark.gpu


def host(t):
    return t.float().cpu().numpy()


def reference_weights(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    ocfg = oracle.m1_config(d_model=128, n_layers=2, d_state=16, d_conv=4, expand=2, dt_rank=8, input_dim=128)
    flat = oracle.m1_weights_init(ocfg, 42)
    lv = oracle.m1_layer_views(ocfg, flat)
    cfg = mb.MambaConfig(d_model=128, n_layers=2, d_state=16, d_conv=4, expand=2, dt_rank=8)
    w = mb.MambaWeights(cfg, cuda_dev, dtype=torch.float32)
    w.load_layers(lv["layers"], lv["norm_f"])
    return ocfg, flat, lv, cfg, w


def test_backbone_prefill_matches_the_cpu_backbone_end_to_end(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    ocfg, flat, lv, cfg, w = reference_weights(cuda_dev)
    B, T = 4, 512
    inp = np.random.default_rng(7).standard_normal((B, T, 128)).astype(np.float32)
    refs = [oracle.m1_prefill(ocfg, flat, inp[b]) for b in range(B)]
    # input projection (a GEMM outside the path) on the host, as the oracle does it
    temporal = (inp.astype(np.float64) @ lv["input_proj_w"].astype(np.float64) + lv["input_proj_b"]).astype(np.float32)
    bb = mb.GpuMambaBackbone(w, B)
    out = bb.prefill_sequence(torch.from_numpy(temporal).to(cuda_dev))
    torch.cuda.synchronize()
    ref_out = np.stack([r["out"] for r in refs])
    assert rel_err(host(out), ref_out) <= 1e-4
    assert rel_err(host(bb.ssm), np.stack([r["ssm_state"] for r in refs], axis=1)) <= 1e-4
    np.testing.assert_allclose(host(bb.conv), np.stack([r["conv_state"] for r in refs], axis=1), rtol=0, atol=2e-5)
    mb.ffi.default_handle(0).check_status()


def test_decode_steps_continue_the_prefill(cuda_dev):
    """prefill(T) followed by step() on the next tokens == prefill(T + k) (tests/prefill.rs:174-232)."""
    import torch

    import mamba_rs_b200 as mb
    _, _, _, cfg, w = reference_weights(cuda_dev)
    B, T, k = 3, 100, 5
    g = torch.Generator(device=cuda_dev).manual_seed(3)
    x = torch.randn(B, T + k, 128, device=cuda_dev, generator=g)
    whole = mb.GpuMambaBackbone(w, B)
    ref = whole.prefill_sequence(x.clone())
    bb = mb.GpuMambaBackbone(w, B)
    head = bb.prefill_sequence(x[:, :T].clone().contiguous())
    steps = [bb.step(x[:, T + i].clone().contiguous()) for i in range(k)]
    torch.cuda.synchronize()
    got = torch.cat([head, torch.stack(steps, dim=1)], dim=1)
    assert rel_err(host(got), host(ref)) <= 1e-4
    assert rel_err(host(bb.ssm), host(whole.ssm)) <= 1e-4
    bb.reset()
    assert float(bb.ssm.abs().max()) == 0.0 and float(bb.conv.abs().max()) == 0.0


def torch_reference_loss(w, cfg, ids):
    """float64 restatement of the training forward with autograd (sequential scan)."""
    import torch
    import torch.nn.functional as F
    P = [{k: v.detach().double().requires_grad_(True) for k, v in w.layer(l, "master").items()} for l in range(cfg.n_layers)]
    tail = {k: v.detach().double().requires_grad_(True) for k, v in w.tail("master").items()}
    B, T1 = ids.shape
    T, di, N, dr, K = T1 - 1, cfg.d_inner, cfg.d_state, cfg.dt_rank, cfg.d_conv
    s = tail["embedding"][ids[:, :-1].long()]

    def norm(x, wt):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + cfg.rms_norm_eps) * wt

    for p in P:
        post = norm(s, p["norm_w"])
        proj = post @ p["in_proj_w"]
        x, z = proj[..., :di], proj[..., di:]
        xp = F.pad(x.transpose(1, 2), (K - 1, 0))
        u = F.silu(F.conv1d(xp, p["conv_w"][:, None, :], p["conv_b"], groups=di)).transpose(1, 2)
        xdbl = u @ p["x_proj_w"]
        delta = F.softplus(xdbl[..., :dr] @ p["dt_proj_w"] + p["dt_proj_b"])
        Bm, Cm = xdbl[..., dr:dr + N], xdbl[..., dr + N:]
        a = -torch.exp(p["a_log"])
        h = torch.zeros(B, di, N, dtype=torch.float64, device=s.device)
        ys = []
        for t in range(T):
            h = torch.exp(delta[:, t, :, None] * a) * h + (delta[:, t] * u[:, t])[..., None] * Bm[:, t, None, :]
            ys.append((h * Cm[:, t, None, :]).sum(-1) + p["d_param"] * u[:, t])
        y = torch.stack(ys, 1) * F.silu(z)
        s = s + y @ p["out_proj_w"]
    logits = norm(s, tail["norm_f"]) @ tail["embedding"].t()
    loss = F.cross_entropy(logits.view(B * T, -1), ids[:, 1:].reshape(-1).long())
    loss.backward()
    return loss.item(), P, tail


def test_training_step_gradients_match_autograd_and_adamw_reduces_the_loss(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    cfg = mb.MambaConfig(d_model=32, n_layers=2, d_state=16, d_conv=4, expand=2)
    V, B, T = 50, 2, 70
    w = mb.MambaWeights(cfg, cuda_dev, dtype=torch.float32, vocab=V).init_random(5)
    ids = torch.randint(0, V, (B, T + 1), device=cuda_dev, dtype=torch.int32,
                        generator=torch.Generator(device=cuda_dev).manual_seed(1))
    tr = mb.MambaLMTrainer(w, lr=3e-3, weight_decay=0.0)
    loss = tr.forward(ids)
    tr.backward_step(accumulate_only=True)
    torch.cuda.synchronize()
    ref_loss, P, tail = torch_reference_loss(w, cfg, ids)
    assert abs(float(loss) - ref_loss) <= 1e-4 * abs(ref_loss)
    for l in range(cfg.n_layers):
        g = w.layer(l, "grad")
        for k, v in P[l].items():
            assert rel_err(host(g[k]), v.grad.cpu().numpy()) <= 2e-3, (l, k)
    gt = w.tail("grad")
    for k, v in tail.items():
        assert rel_err(host(gt[k]), v.grad.cpu().numpy()) <= 2e-3, k
    # a few optimiser steps on the same batch: the loss goes down
    w.grad.zero_()
    tr._pending = 0
    first = float(tr.step(ids))
    for _ in range(5):
        last = float(tr.step(ids))
    assert last < first
    mb.ffi.default_handle(0).check_status()


def test_bf16_training_step_runs_at_a_model_layer_shape(cuda_dev):
    """130m layer shape (d_model 768, d_inner 1536, dt_rank 48), 2 layers, bf16: finite loss
    close to ln(vocab) at initialisation, finite gradients."""
    import torch

    import mamba_rs_b200 as mb
    cfg = mb.MambaConfig(d_model=768, n_layers=2)
    V, B, T = 5000, 2, 256
    w = mb.MambaWeights(cfg, cuda_dev, dtype=torch.bfloat16, vocab=V).init_random(0)
    ids = torch.randint(0, V, (B, T + 1), device=cuda_dev, dtype=torch.int32)
    tr = mb.MambaLMTrainer(w)
    loss = tr.forward(ids)
    tr.backward_step(accumulate_only=True)
    torch.cuda.synchronize()
    assert abs(float(loss) - np.log(V)) < 0.5
    assert bool(torch.isfinite(w.grad).all()) and float(w.grad.abs().max()) > 0


def test_greedy_decode_from_a_captured_graph_equals_eager_decode(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    from mamba_rs_b200 import model
    cfg = mb.MambaConfig(d_model=128, n_layers=3)
    V, B, T, n = 997, 4, 60, 12
    w = mb.MambaWeights(cfg, cuda_dev, dtype=torch.bfloat16, vocab=V).init_random(11)
    ids = torch.randint(0, V, (B, T), device=cuda_dev, dtype=torch.int32,
                        generator=torch.Generator(device=cuda_dev).manual_seed(2))
    outs = []
    for use_graph in (False, True):
        lm = mb.GpuMambaLM(w, B)
        lm.prefill(ids)
        lm._dec = model._DecodePlan(lm.backbone, B, lm)
        lm._dec.ok = lm.backbone._plan(B).ok = False  # (the one-launch kernel would take both)
        outs.append(lm.generate_greedy(n, use_graph=use_graph).cpu().numpy())
        assert (lm._graph is not None) == use_graph
    np.testing.assert_array_equal(outs[0], outs[1])
    assert outs[0].min() >= 0 and outs[0].max() < V


@pytest.mark.parametrize("dt", ["bf16", "f32"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 33, 2), (3, 130, 2)], ids=lambda s: "b%dt%dl%d" % s)
def test_passes_that_come_again_equal_the_first_ones(cuda_dev, shape, dt):
    """From the third call with the same addresses on a pass is a replay; other ids, other lengths in
    between, a result that the caller keeps and changed hyperparameters give what single launches give."""
    import torch

    import mamba_rs_b200 as mb
    B, T, L = shape
    td = {"bf16": torch.bfloat16, "f32": torch.float32}[dt]
    make = lambda: mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=L), cuda_dev, dtype=td, vocab=300).init_random(3)  # noqa: E731
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    ids = [torch.randint(0, 300, (B, T + 1), device=cuda_dev, dtype=torch.int32, generator=g) for _ in range(6)]
    x = torch.randn(B, T, 64, device=cuda_dev, generator=g)
    runs = []
    for replay in (False, True):
        w, got = make(), []
        lm = mb.GpuMambaLM(w, B)
        for (n, i) in ((T, 0), (T, 1), (T, 2), (T + 1, 3), (T, 4), (T, 5)):
            lm.backbone._prefill_plan(B, n).launch_bound = replay
            lm.backbone.reset()
            got += [lm.prefill(ids[i][:, :n]).clone(), lm.next_ids.clone(), lm.backbone.ssm.clone(), lm.backbone.conv.clone()]
        buf, kept = torch.empty_like(x), []
        for i in range(5):
            lm.backbone.reset()
            buf.copy_(x * (i + 1))
            kept.append(lm.backbone.prefill_sequence(buf))
            got.append(buf.clone())
        got += kept
        tr = mb.MambaLMTrainer(w, lr=1e-3)
        tr._plan(B, T).launch_bound = replay
        for i in range(6):
            if i == 4:
                tr.lr = 2e-3
            got.append(tr.step(ids[i]))
        got += [w.master.clone(), w.lp.clone(), tr.m, tr.v]
        assert bool(lm.backbone._prefill_plan(B, T).replay.kept) == replay == bool(tr._plan(B, T).replay.kept)
        runs.append(got)
    for a, b in zip(*runs):
        assert rel_err(b.float().cpu().numpy(), a.float().cpu().numpy()) <= (1e-5 if dt == "f32" else 2e-2)
    mb.ffi.default_handle(0).check_status()


def test_steps_by_operators_that_come_again_equal_the_first_ones(cuda_dev):
    """A model the one-launch step does not take (d_state 8): the third step with the same rows is a replay."""
    import torch

    import mamba_rs_b200 as mb
    w = mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=2, d_state=8), cuda_dev, dtype=torch.float32).init_random(3)
    again, once = mb.GpuMambaBackbone(w, 3), mb.GpuMambaBackbone(w, 3)
    assert not again._plan(3).ok
    buf, xs = torch.empty(3, 64, device=cuda_dev), torch.randn(6, 3, 64, device=cuda_dev)
    got = []
    for x in xs:
        buf.copy_(x)
        got.append((again.step(buf), buf.clone()))
    assert again._plan(3).replay.kept
    for x, (out, res) in zip(xs, got):
        once._plan(3).replay.seen.clear()
        y = x.clone()
        ref = once.step(y)
        assert rel_err(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-6 and rel_err(res.cpu().numpy(), y.cpu().numpy()) <= 1e-6
    assert not once._plan(3).replay.kept and torch.equal(again.ssm, once.ssm) and torch.equal(again.conv, once.conv)


def test_an_engine_made_on_a_device_by_name(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    w = mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=1), "cuda", vocab=50).init_random(3)
    lm, ids = mb.GpuMambaLM(w, 2), torch.randint(0, 50, (2, 9), device=cuda_dev, dtype=torch.int32)
    for _ in range(4):
        assert bool(torch.isfinite(lm.prefill(ids).float()).all())
    assert lm.generate_greedy(3).shape == (2, 3)
    assert np.isfinite(float(mb.MambaLMTrainer(w).step(ids)))


@pytest.mark.parametrize("N", [16, 8])  # the one-launch kernel, and operators that are replayed
def test_a_step_follows_replaced_decay_rates_and_a_changed_epsilon(cuda_dev, N):
    import torch

    import mamba_rs_b200 as mb
    make = lambda: mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=2, d_state=N), cuda_dev, dtype=torch.float32).init_random(3)  # noqa: E731
    bb = mb.GpuMambaBackbone(make(), 3)
    buf, x = torch.empty(3, 64, device=cuda_dev), torch.randn(3, 64, device=cuda_dev)

    def run(b, n=4):
        b.reset()
        b.ssm.fill_(0.3)
        for _ in range(n):
            buf.copy_(x)
            out = b.step(buf)
        return out
    run(bb)
    bb.w.a_neg[1] = 3 * bb.w.a_neg[1].clone()
    bb.cfg.rms_norm_eps = 0.5
    fresh = mb.GpuMambaBackbone(make(), 3)
    fresh.w.a_neg[1].mul_(3)
    fresh.cfg.rms_norm_eps = 0.5
    fresh._plan(3).ok = False
    got, want = run(bb), run(fresh, 2)
    want = run(fresh)
    assert rel_err(got.cpu().numpy(), want.cpu().numpy()) <= 1e-5
    assert rel_err(bb.ssm.cpu().numpy(), fresh.ssm.cpu().numpy()) <= 1e-5


def test_prefill_and_training_follow_a_changed_epsilon(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    make = lambda: mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=2), cuda_dev, dtype=torch.float32, vocab=50).init_random(3)  # noqa: E731
    ids = torch.randint(0, 50, (2, 21), device=cuda_dev, dtype=torch.int32)
    lm, ref = mb.GpuMambaLM(make(), 2), mb.GpuMambaLM(make(), 2)
    tr, tref = mb.MambaLMTrainer(make()), mb.MambaLMTrainer(make())
    for _ in range(4):
        lm.backbone.reset()
        lm.prefill(ids)
        tr.step(ids)
        tref.step(ids)
    for c in (lm.w.cfg, ref.w.cfg, tr.cfg, tref.cfg):
        c.rms_norm_eps = 0.5
    lm.backbone.reset()
    assert rel_err(lm.prefill(ids).cpu().numpy(), ref.prefill(ids).cpu().numpy()) <= 1e-6
    tref._plan(2, 20).launch_bound = False
    assert abs(float(tr.step(ids)) - float(tref.step(ids))) <= 1e-6


def test_what_a_capture_makes_serves_no_later_call(cuda_dev):
    """The first call of an engine inside a capture: its workspaces are filled by the graph's replays alone, so
    an eager call before the first replay makes its own."""
    import torch

    import mamba_rs_b200 as mb
    make = lambda: mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=2), cuda_dev, dtype=torch.float32, vocab=50).init_random(3)  # noqa: E731
    x, ids = torch.randn(3, 64, device=cuda_dev), torch.randint(0, 50, (3, 9), device=cuda_dev, dtype=torch.int32)
    warm, wt = mb.GpuMambaLM(make(), 3), mb.MambaLMTrainer(make())
    want_step = warm.backbone.step(x.clone())  # (and kernels are loaded)
    warm.backbone.reset()
    want = warm.generate_greedy(3), warm.backbone.ssm.clone()
    want_loss = wt.forward(ids)
    wt.backward_step(accumulate_only=True)
    lm, tr = mb.GpuMambaLM(make(), 3), mb.MambaLMTrainer(make())
    bb = mb.GpuMambaBackbone(lm.w, 3)
    bufs, graph = torch.empty(3, 64, device=cuda_dev), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = bb.step(bufs)
        toks = lm.generate_greedy(3)
        loss = tr.forward(ids)
        tr.backward_step(accumulate_only=True)
    assert not bb._plans and lm._dec is None and not tr._plans
    for again in (False, True):
        bb.reset(), lm.backbone.reset()
        lm.next_ids.zero_(), tr.w.grad.zero_()
        if not again:
            assert torch.equal(bb.step(x.clone()), want_step)
            assert torch.equal(lm.generate_greedy(3), want[0]) and torch.equal(lm.backbone.ssm, want[1])
        else:
            bufs.copy_(x)
            graph.replay()
            assert torch.equal(out, want_step) and torch.equal(toks, want[0]) and torch.equal(lm.backbone.ssm, want[1])
            assert float(loss) == float(want_loss)
            assert rel_err(tr.w.grad.cpu().numpy(), wt.w.grad.cpu().numpy()) <= 1e-6
    mb.ffi.default_handle(0).check_status()


def test_input_buffers_in_rotation_are_right_and_record_a_bounded_number_of_times(cuda_dev, monkeypatch):
    import torch

    import mamba_rs_b200 as mb
    from mamba_rs_b200 import model
    monkeypatch.setattr(model._Shelf, "KEEP", 3)
    recorded = []
    record = model._Shelf.record
    monkeypatch.setattr(model._Shelf, "record", lambda self, launch: recorded.append(1) or record(self, launch))
    w = mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=2), cuda_dev, dtype=torch.float32).init_random(3)
    bb, one = mb.GpuMambaBackbone(w, 2), mb.GpuMambaBackbone(w, 2)
    one._prefill_plan(2, 20).launch_bound = False
    x = torch.randn(2, 20, 64, device=cuda_dev)
    bufs = [torch.empty_like(x) for _ in range(7)]
    for i in range(10):
        for b in bufs:
            for e in (bb, one):
                e.reset()
            b.copy_(x * (i + 1))
            got = bb.prefill_sequence(b)
            want = one.prefill_sequence(x * (i + 1))
            assert torch.equal(got, want)
    assert len(recorded) == 3 == len(bb._prefill_plan(2, 20).replay.kept)


def test_a_learning_rate_schedule_keeps_the_recorded_step(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    make = lambda: mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=2), cuda_dev, dtype=torch.float32, vocab=50).init_random(3)  # noqa: E731
    ids = torch.randint(0, 50, (2, 21), device=cuda_dev, dtype=torch.int32)
    tr, ref = mb.MambaLMTrainer(make()), mb.MambaLMTrainer(make())
    ref._plan(2, 20).launch_bound = False
    for i in range(8):
        for t in (tr, ref):
            t.lr, t.wd = 1e-3 * (i + 1) / 8, 0.1 / (i + 1)
        assert abs(float(tr.step(ids)) - float(ref.step(ids))) <= 1e-5
    assert len(tr._plan(2, 20).replay.kept) == 1 and tr.t == ref.t == 8 and not ref._plan(2, 20).replay.kept
    for a, b in ((tr.w.master, ref.w.master), (tr.m, ref.m), (tr.v, ref.v)):
        assert rel_err(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5


def test_a_step_that_fails_leaves_the_step_count(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    w = mb.MambaWeights(mb.MambaConfig(d_model=64, n_layers=1), cuda_dev, dtype=torch.float32, vocab=50).init_random(3)
    tr, ids = mb.MambaLMTrainer(w), torch.randint(0, 50, (1, 9), device=cuda_dev, dtype=torch.int32)
    forward = tr.forward
    for i in range(5):  # (the third would be recorded)
        def fail(ids):
            forward(ids)
            raise torch.OutOfMemoryError("no room")
        tr.forward = fail
        with pytest.raises(torch.OutOfMemoryError):
            tr.step(ids)
        tr._acts = None
        assert tr.t == 0 and not tr._plan(1, 8).replay.kept
    tr.forward = forward
    assert np.isfinite(float(tr.step(ids))) and tr.t == 1


def test_greedy_decode_by_operators_eager_captured_and_the_one_launch_kernel_agree(cuda_dev):
    """The three ways generate_greedy has: operators launched one by one (use_graph=False), the captured step
    where the kernel does not take the model, and the kernel."""
    import torch

    import mamba_rs_b200 as mb
    from mamba_rs_b200 import model
    w = mb.MambaWeights(mb.MambaConfig(d_model=128, n_layers=3), cuda_dev, vocab=997).init_random(11)
    w.tail("master")["embedding"].mul_(50.0)
    w.refresh()
    ids = torch.randint(0, 997, (4, 60), device=cuda_dev, dtype=torch.int32, generator=torch.Generator(device=cuda_dev).manual_seed(2))
    got = {}
    for way in ("eager", "captured", "kernel"):
        lm = mb.GpuMambaLM(w, 4)
        lm.prefill(ids)
        lm._dec = model._DecodePlan(lm.backbone, 4, lm)
        if way == "captured":
            lm._dec.ok = False
            lm.backbone._plan(4).ok = False
        before = lm._dec.ws[:4].view(torch.int32).item()
        got[way] = lm.generate_greedy(12, use_graph=way != "eager").cpu().numpy(), lm.backbone.ssm.cpu().numpy()
        assert (lm._graph is not None) == (way == "captured")
        assert (lm._dec.ws[:4].view(torch.int32).item() > before) == (way == "kernel")  # tags used by launches
        assert lm.backbone._plan(4).ok == (way != "captured") and (way == "kernel" or not int(lm.backbone._plan(4).ws[:4].view(torch.int32)))
    np.testing.assert_array_equal(got["eager"][0], got["captured"][0])
    np.testing.assert_array_equal(got["eager"][1], got["captured"][1])
    np.testing.assert_array_equal(got["kernel"][0], got["eager"][0])
    assert rel_err(got["kernel"][1], got["eager"][1]) <= 2e-2


def test_a_workspace_is_not_handed_on_while_another_stream_uses_it(cuda_dev):
    """A step on a stream that is held up, its plan dropped meanwhile: memory asked for on the plan's own stream
    must not be the workspace that the step has yet to use."""
    import torch

    import mamba_rs_b200 as mb
    w = mb.MambaWeights(mb.MambaConfig(d_model=256, n_layers=2), cuda_dev).init_random(3)
    bb, side = mb.GpuMambaBackbone(w, 16), torch.cuda.Stream(device=cuda_dev)
    x = torch.randn(16, 256, device=cuda_dev)
    want = bb.step(x.clone())
    for again in (False, True):
        bb.reset()
        y, held = x.clone(), bb._plan(16).ws
        at, size = held.data_ptr(), held.numel()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(50_000_000)
            got = bb.step(y)
        del held
        bb._plans.clear()
        taken = [torch.full((size,), 255, dtype=torch.uint8, device=cuda_dev) for _ in range(4)]
        assert at not in [t.data_ptr() for t in taken]
        side.synchronize()
        assert torch.equal(got, want)
        del taken

def test_one_launch_steps_from_the_start_match_the_cpu_backbone(cuda_dev):
    """Every step of a sequence by the whole-model decode launch, against the CPU oracle's token loop."""
    import torch

    import mamba_rs_b200 as mb
    ocfg, flat, lv, _, w = reference_weights(cuda_dev)
    B, T = 3, 40
    inp = np.random.default_rng(9).standard_normal((B, T, 128)).astype(np.float32)
    refs = [oracle.m1_prefill(ocfg, flat, inp[b]) for b in range(B)]
    temporal = (inp.astype(np.float64) @ lv["input_proj_w"].astype(np.float64) + lv["input_proj_b"]).astype(np.float32)
    bb = mb.GpuMambaBackbone(w, B)
    assert bb._plan(B).ok
    outs = [bb.step(torch.from_numpy(np.ascontiguousarray(temporal[:, t])).to(cuda_dev)) for t in range(T)]
    got = torch.stack(outs, 1)
    assert rel_err(host(got), np.stack([r["out"] for r in refs])) <= 1e-4
    assert rel_err(host(bb.ssm), np.stack([r["ssm_state"] for r in refs], axis=1)) <= 1e-4
    np.testing.assert_allclose(host(bb.conv), np.stack([r["conv_state"] for r in refs], axis=1), rtol=0, atol=2e-5)
    mb.ffi.default_handle(0).check_status()
