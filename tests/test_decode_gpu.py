"""The whole-model decode launch (csrc/decode.cu) against the same step made of the library's
operators one by one, at sizes where its split over CTAs, tiles, K slices and batch passes changes."""
import numpy as np
import pytest

from helpers import rel_err, torch_dtype

pytestmark = pytest.mark.gpu

# d_model, layers, batch: one tile per CTA and less, ragged K slices (d_model 8, 72, 200), more than one
# batch pass (9 in f32, 17 and 40), the widest model and batch it takes
SIZES = [(128, 3, 1), (8, 2, 3), (72, 2, 9), (200, 2, 17), (768, 2, 8), (1024, 1, 40), (64, 2, 64)]


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "d%dl%db%d" % s)
def test_one_launch_step_matches_the_operators(cuda_dev, size, dt):
    import torch

    import mamba_rs_b200 as mb
    d, L, B = size
    w = mb.MambaWeights(mb.MambaConfig(d_model=d, n_layers=L), cuda_dev, dtype=torch_dtype(dt)).init_random(3)
    g = torch.Generator(device=cuda_dev).manual_seed(B)
    fast, slow = mb.GpuMambaBackbone(w, B), mb.GpuMambaBackbone(w, B)
    slow._plan(B).ok = False
    # (f32 at 1024: its tiles, 2 x 4 of 1024 rows and 2 of 2048, leave too little shared memory for the operand rows)
    assert fast._plan(B).ok == (not (dt == "f32" and d == 1024))
    for bb in (fast, slow):
        g2 = torch.Generator(device=cuda_dev).manual_seed(7)
        bb.conv.copy_(torch.randn(bb.conv.shape, device=cuda_dev, generator=g2))
        bb.ssm.copy_(torch.randn(bb.ssm.shape, device=cuda_dev, generator=g2))
    tol = {"f32": 1e-5, "f16": 4e-3, "bf16": 2e-2}[dt]
    h = lambda t: t.float().cpu().numpy()
    for _ in range(3):
        x = torch.randn(B, d, device=cuda_dev, generator=g)
        xa, xb = x.clone(), x.clone()
        a, b = fast.step(xa), slow.step(xb)
        assert rel_err(h(a), h(b)) <= tol
        assert rel_err(h(xa), h(xb)) <= tol
    assert rel_err(h(fast.conv), h(slow.conv)) <= tol
    assert rel_err(h(fast.ssm), h(slow.ssm)) <= tol
    mb.ffi.default_handle(0).check_status()


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("size", [(128, 2, 1, 997), (72, 1, 9, 50), (256, 2, 17, 5003), (64, 1, 33, 17)],
                         ids=lambda s: "d%dl%db%dv%d" % s)
def test_one_launch_greedy_decode_matches_the_operators(cuda_dev, size, dt):
    import torch

    import mamba_rs_b200 as mb
    d, L, B, V = size
    w = mb.MambaWeights(mb.MambaConfig(d_model=d, n_layers=L), cuda_dev, dtype=torch_dtype(dt), vocab=V).init_random(5)
    w.tail("master")["embedding"].mul_(50.0)  # logits whose order does not hang on a rounding
    w.refresh()
    ids = torch.randint(0, V, (B, 20), device=cuda_dev, dtype=torch.int32,
                        generator=torch.Generator(device=cuda_dev).manual_seed(1))
    got = []
    for fast in (True, False):
        lm = mb.GpuMambaLM(w, B)
        lm.prefill(ids)
        if not fast:
            lm.generate_greedy(0)
            lm._dec.ok = False
        toks = lm.generate_greedy(4)
        assert not fast or lm._dec.ok
        got.append((toks.cpu().numpy(), lm.logits.float().cpu().numpy(), lm.next_ids.cpu().numpy(),
                    lm.backbone.ssm.cpu().numpy()))
        assert np.array_equal(lm.next_ids.cpu().numpy(), lm.logits.argmax(1).cpu().numpy())
    tol = {"f32": 1e-5, "f16": 4e-3, "bf16": 2e-2}[dt]
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][2], got[1][2])
    assert rel_err(got[0][1], got[1][1]) <= tol
    assert rel_err(got[0][3], got[1][3]) <= tol
    mb.ffi.default_handle(0).check_status()


def filled(bb, seed):
    import torch
    g = torch.Generator(device=bb.conv.device).manual_seed(seed)
    bb.conv.copy_(torch.randn(bb.conv.shape, device=bb.conv.device, generator=g))
    bb.ssm.copy_(torch.randn(bb.ssm.shape, device=bb.conv.device, generator=g))
    return torch.randn(bb.batch, bb.cfg.d_model, device=bb.conv.device, generator=g)


@pytest.mark.parametrize("dt,d,L,B", [("bf16", 128, 3, 4), ("f32", 256, 2, 3), ("bf16", 768, 2, 20)])
def test_a_step_after_one_that_gave_up_is_right(cuda_dev, dt, d, L, B):
    """A launch whose waits may take one poll gives up, says so, and leaves a workspace that the next launch
    can use: no word of the one that failed may pass for its own."""
    import torch

    import mamba_rs_b200 as mb
    h = mb.ffi.default_handle(0)
    h.check_status()
    w = mb.MambaWeights(mb.MambaConfig(d_model=d, n_layers=L), cuda_dev, dtype=torch_dtype(dt)).init_random(3)
    bb, ref = mb.GpuMambaBackbone(w, B), mb.GpuMambaBackbone(w, B)
    ctl = bb._plan(B).ws[:16].view(torch.int32)
    for n in range(1, 4):
        x = filled(bb, n)
        ctl[2] = 1
        bb.step(x)
        with pytest.raises(RuntimeError, match="bounded wait"):
            h.check_status()
        assert ctl.tolist()[:2] == [(2 * n - 1) * (L + 2), 0]
        ctl[2] = 0
        x = filled(bb, 10 + n)
        want = ref.step(filled(ref, 10 + n))
        got = bb.step(x)
        assert torch.equal(got, want) and torch.equal(bb.ssm, ref.ssm) and torch.equal(bb.conv, ref.conv)
        h.check_status()
        assert ctl.tolist()[:2] == [2 * n * (L + 2), 0]


def test_a_workspace_passes_from_one_batch_size_to_another(cuda_dev):
    """The same memory for 9, 2 and 9 sequences without clearing, then cleared and used again."""
    import torch

    import mamba_rs_b200 as mb
    w = mb.MambaWeights(mb.MambaConfig(d_model=128, n_layers=2), cuda_dev).init_random(3)
    big, small = mb.GpuMambaBackbone(w, 9), mb.GpuMambaBackbone(w, 2)
    ws = big._plan(9).ws
    small._plan(2).ws = ws
    small._plan(2).args.workspace = ws.data_ptr()
    for n, bb in enumerate((big, small, big, small)):
        if n == 3:
            ws.zero_()
        ref = mb.GpuMambaBackbone(w, bb.batch)
        want = ref.step(filled(ref, n))
        got = bb.step(filled(bb, n))
        assert torch.equal(got, want) and torch.equal(bb.ssm, ref.ssm)
    mb.ffi.default_handle(0).check_status()
