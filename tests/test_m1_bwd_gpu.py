"""GPU parity tests of the fused Mamba-1 backward (BPTT by recomputation)
against the CPU oracle's analytic backward on identical inputs.

Bar: max-abs error / max-abs reference <= 1e-4 (f32 storage) or 2e-2 (bf16 /
f16 storage) per gradient tensor; dB, dC, dA_log, dD are f32 accumulators and
are held to 1e-4 / 2e-2 as well (their inputs d_y etc. are storage-rounded)."""
import numpy as np
import pytest

import oracle
from helpers import GOLDEN_CASES, TOL, golden_inputs, load_golden, quantised_inputs, random_states, rel_err, to_dev, torch_dtype
from mamba_rs_b200 import synth

pytestmark = pytest.mark.gpu


def gpu_fwd_bwd(q, dg, dt, dev, ssm0, S, delta_softplus=True):
    import torch

    import mamba_rs_b200 as mb
    td = torch_dtype(dt)
    B, T, D = q["delta_raw"].shape
    N = q["a_neg"].shape[1]
    x, dl, Bm, Cm = [to_dev(q[k], dev, td) for k in ("x", "delta_raw", "Bm", "Cm")]
    z = to_dev(q.get("z"), dev, td)
    a, Dp = to_dev(q["a_neg"], dev), to_dev(q["Dp"], dev)
    cs = torch.empty(B, (T + S - 1) // S, D, N, device=dev)
    ssm = to_dev(ssm0, dev)
    mb.selective_scan_fwd(x, dl, Bm, Cm, a, Dp, z, ssm_state=ssm, chunk_states=cs, save_stride=S,
                          delta_softplus=delta_softplus)
    g = mb.selective_scan_bwd(x, dl, Bm, Cm, a, Dp, to_dev(dg, dev, td), cs, S, z,
                              delta_softplus=delta_softplus)
    torch.cuda.synchronize()
    mb.ffi.default_handle(0).check_status()
    return {k: (None if v is None else v.float().cpu().numpy()) for k, v in g.items()}


SHAPES = [(2, 40, 64, 16), (1, 1, 32, 16), (1, 15, 33, 16), (1, 17, 7, 16), (2, 64, 32, 16),
          (1, 65, 40, 16), (3, 100, 20, 8), (1, 130, 12, 4), (1, 50, 12, 12), (2, 200, 96, 16),
          # d_state > 16: the wide-state kernel (4 ... 32 lanes per channel)
          (2, 70, 20, 32), (1, 100, 9, 64), (1, 40, 5, 24), (1, 33, 3, 128), (1, 65, 2, 256)]


@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("a_mode", ["s4d", "random"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B%dT%dD%dN%d" % s)
def test_fused_backward_matches_oracle(cuda_dev, shape, a_mode, dt):
    B, T, D, N = shape
    q = quantised_inputs(B, T, D, N, 0, dt, seed=B * 100 + T, a_mode=a_mode)
    ssm0, _ = random_states(B, D, N, 0, seed=T + 1)
    dg = synth.round_to(np.random.default_rng(T).standard_normal((B, T, D)).astype(np.float32), dt)
    ref = oracle.m1_fused_bwd(q["x"], q["delta_raw"], q["Bm"], q["Cm"], q["z"], q["a_neg"], q["Dp"], dg,
                              ssm_state0=ssm0)
    S = 64 if T % 3 else 32
    g = gpu_fwd_bwd(q, dg, dt, cuda_dev, ssm0, S)
    tol = TOL[dt]
    assert rel_err(g["d_u"], ref["d_x"]) <= tol
    assert rel_err(g["d_delta"], ref["d_delta"]) <= tol
    assert rel_err(g["d_z"], ref["d_z"]) <= tol
    for k in ("dB", "dC", "dA_log", "dD"):
        assert rel_err(g[k], ref[k]) <= max(tol, 2e-4), k


@pytest.mark.parametrize("S", [32, 64])
def test_every_save_stride(cuda_dev, S):
    q = quantised_inputs(2, 150, 32, 16, 0, "f32", seed=S)
    dg = np.random.default_rng(S).standard_normal((2, 150, 32)).astype(np.float32)
    ref = oracle.m1_fused_bwd(q["x"], q["delta_raw"], q["Bm"], q["Cm"], q["z"], q["a_neg"], q["Dp"], dg)
    g = gpu_fwd_bwd(q, dg, "f32", cuda_dev, np.zeros((2, 32, 16), np.float32), S)
    for gk, rk in (("d_u", "d_x"), ("d_delta", "d_delta"), ("d_z", "d_z"), ("dB", "dB"), ("dC", "dC"),
                   ("dA_log", "dA_log"), ("dD", "dD")):
        assert rel_err(g[gk], ref[rk]) <= 2e-4, gk


@pytest.mark.parametrize("case", [c for c in GOLDEN_CASES if c[5] == 0], ids=lambda c: c[0])
def test_fused_backward_matches_golden(cuda_dev, case):
    q, ssm0, _, dg = golden_inputs(case)
    gold = load_golden(case[0])
    dt = case[6]
    g = gpu_fwd_bwd(q, synth.round_to(dg, dt), dt, cuda_dev, ssm0, 32)
    # the fixture's upstream gradient is unrounded f32; compare within the storage tolerance
    assert rel_err(g["d_u"], gold["d_x"]) <= TOL[dt]
    assert rel_err(g["dB"], gold["dB"]) <= TOL[dt]
    assert rel_err(g["dA_log"], gold["dA_log"]) <= TOL[dt]


def test_backward_without_gate_and_without_softplus(cuda_dev):
    q = quantised_inputs(2, 70, 24, 16, 0, "f32", seed=9, a_mode="random")
    q["delta_raw"] = np.log1p(np.exp(q["delta_raw"].astype(np.float64))).astype(np.float32)
    q["z"] = None
    dg = np.random.default_rng(1).standard_normal((2, 70, 24)).astype(np.float32)
    ref = oracle.m1_fused_bwd(q["x"], q["delta_raw"], q["Bm"], q["Cm"], None, q["a_neg"], q["Dp"], dg,
                              delta_softplus=False)
    g = gpu_fwd_bwd(q, dg, "f32", cuda_dev, np.zeros((2, 24, 16), np.float32), 64, delta_softplus=False)
    assert g["d_z"] is None
    for gk, rk in (("d_u", "d_x"), ("d_delta", "d_delta"), ("dB", "dB"), ("dC", "dC"),
                   ("dA_log", "dA_log"), ("dD", "dD")):
        assert rel_err(g[gk], ref[rk]) <= 2e-4, gk


def test_parameter_gradients_accumulate_and_are_reproducible(cuda_dev):
    """dA_log / dD are '+=' (grad-arena convention) and the two-stage
    reductions are atomics-free: two runs give identical bits."""
    import torch
    q = quantised_inputs(3, 90, 40, 16, 0, "bf16", seed=4)
    dg = synth.round_to(np.random.default_rng(2).standard_normal((3, 90, 40)).astype(np.float32), "bf16")
    z0 = np.zeros((3, 40, 16), np.float32)
    g1 = gpu_fwd_bwd(q, dg, "bf16", cuda_dev, z0, 64)
    g2 = gpu_fwd_bwd(q, dg, "bf16", cuda_dev, z0, 64)
    for k in ("d_u", "d_delta", "d_z", "dB", "dC", "dA_log", "dD"):
        np.testing.assert_array_equal(g1[k], g2[k])


def test_backward_full_size_config2_properties(cuda_dev):
    """Config #2 at full size: gradients are linear in dy (scale by 2 exactly,
    a power of two), finite, and a 2-channel slice matches the oracle."""
    import torch

    import mamba_rs_b200 as mb
    B, T, D, N, S = 16, 2048, 1536, 16, 64
    inp = synth.m1_scan_inputs(B, T, D, N, 0, seed=3, a_mode="s4d")
    td = torch.bfloat16
    x, dl, Bm, Cm, z = [to_dev(inp[k], cuda_dev, td) for k in ("x", "delta_raw", "Bm", "Cm", "z")]
    a, Dp = to_dev(inp["a_neg"], cuda_dev), to_dev(inp["Dp"], cuda_dev)
    dy = to_dev(np.random.default_rng(5).standard_normal((B, T, D)).astype(np.float32), cuda_dev, td)
    cs = torch.empty(B, T // S, D, N, device=cuda_dev)
    mb.selective_scan_fwd(x, dl, Bm, Cm, a, Dp, z, chunk_states=cs, save_stride=S)
    g1 = mb.selective_scan_bwd(x, dl, Bm, Cm, a, Dp, dy, cs, S, z)
    g2 = mb.selective_scan_bwd(x, dl, Bm, Cm, a, Dp, dy * 2, cs, S, z)
    torch.cuda.synchronize()
    for k in ("d_u", "d_delta", "d_z", "dB", "dC", "dA_log", "dD"):
        assert torch.isfinite(g1[k].float()).all()
        assert torch.equal(g2[k].float(), 2 * g1[k].float()), k
    bsel, dsel = 3, [5, 1000]
    f = lambda t_: t_[bsel:bsel + 1].float().cpu().numpy()
    # dB/dC need every channel; check the per-channel gradients on the slice
    ref = oracle.m1_fused_bwd(f(x)[..., dsel], f(dl)[..., dsel], f(Bm), f(Cm), f(z)[..., dsel],
                              inp["a_neg"][dsel], inp["Dp"][dsel], f(dy)[..., dsel])
    assert rel_err(f(g1["d_u"])[..., dsel], ref["d_x"]) <= TOL["bf16"]
    assert rel_err(f(g1["d_delta"])[..., dsel], ref["d_delta"]) <= TOL["bf16"]
    assert rel_err(f(g1["d_z"])[..., dsel], ref["d_z"]) <= TOL["bf16"]


# few (sample, channel tile) pairs: the blocks are split into time segments with an exact carry of dh;
# lengths around whole segments and blocks, an unaligned channel count, both save strides
SEG_SHAPES = [(1, 64, 16, 16), (1, 129, 24, 16), (1, 1030, 16, 12), (2, 700, 33, 16), (1, 4100, 8, 16)]


@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("S", [32, 64])
@pytest.mark.parametrize("shape", SEG_SHAPES, ids=lambda s: "B%dT%dD%dN%d" % s)
def test_time_segments_of_the_backward_match_oracle(cuda_dev, shape, S, dt):
    B, T, D, N = shape
    q = quantised_inputs(B, T, D, N, 0, dt, seed=T, a_mode="random" if T % 2 else "s4d")
    ssm0, _ = random_states(B, D, N, 0, seed=T + 1)
    dg = synth.round_to(np.random.default_rng(T).standard_normal((B, T, D)).astype(np.float32), dt)
    ref = oracle.m1_fused_bwd(q["x"], q["delta_raw"], q["Bm"], q["Cm"], q["z"], q["a_neg"], q["Dp"], dg, ssm_state0=ssm0)
    g = gpu_fwd_bwd(q, dg, dt, cuda_dev, ssm0, S)
    for gk, rk in (("d_u", "d_x"), ("d_delta", "d_delta"), ("d_z", "d_z"), ("dB", "dB"), ("dC", "dC"),
                   ("dA_log", "dA_log"), ("dD", "dD")):
        assert rel_err(g[gk], ref[rk]) <= TOL[dt], gk


@pytest.mark.parametrize("D", [16, 40, 400])  # one channel tile, fewer tiles than warps of a value, more
def test_sums_over_channel_tiles_of_small_and_large_calls_agree(cuda_dev, D):
    """dB and dC of five samples at once (a thread a value) and one by one (eight warps a value)."""
    import torch

    B, T = 5, 2048
    q = quantised_inputs(B, T, D, 16, 0, "f32", seed=D)
    dg = np.random.default_rng(D).standard_normal((B, T, D)).astype(np.float32)
    ssm0, _ = random_states(B, D, 16, 0, seed=D)
    whole = gpu_fwd_bwd(q, dg, "f32", cuda_dev, ssm0, 32)
    for b in range(B):
        one = {k: (v[b:b + 1] if k in ("x", "delta_raw", "Bm", "Cm", "z") else v) for k, v in q.items()}
        g = gpu_fwd_bwd(one, dg[b:b + 1], "f32", cuda_dev, ssm0[b:b + 1], 32)
        for k in ("dB", "dC"):
            assert rel_err(g[k][0], whole[k][b]) <= 1e-5
    torch.cuda.synchronize()


@pytest.mark.parametrize("dt", ["f32", "bf16"])
def test_a_workspace_for_a_larger_batch_serves_a_smaller_one(cuda_dev, dt):
    """22 sequences are cut into time segments and would take more than 23, which are not: with the memory of
    23 they run in fewer segments."""
    import torch

    import mamba_rs_b200 as mb
    B, T, D, N, S = 22, 128, 640, 16, 32
    size = mb.selective_scan_bwd_workspace_bytes
    assert size(B, T, D, N) > size(B + 1, T, D, N)
    q = quantised_inputs(B, T, D, N, 0, dt, seed=1)
    td = torch_dtype(dt)
    t = lambda k, d=None: to_dev(q[k], cuda_dev, d)  # noqa: E731
    args = [t("x", td), t("delta_raw", td), t("Bm", td), t("Cm", td), t("a_neg"), t("Dp")]
    z, dy = t("z", td), torch.randn(B, T, D, device=cuda_dev, generator=torch.Generator(device=cuda_dev).manual_seed(2)).to(td)
    cs = torch.empty(B, T // S, D, N, device=cuda_dev)
    mb.selective_scan_fwd(*args, z, chunk_states=cs, save_stride=S)
    run = lambda n: mb.selective_scan_bwd(*args, dy, cs, S, z, workspace=torch.empty(n, dtype=torch.uint8, device=cuda_dev))  # noqa: E731
    own, lent = run(size(B, T, D, N)), run(size(B + 1, T, D, N))
    for k in own:
        assert rel_err(lent[k].float().cpu().numpy(), own[k].float().cpu().numpy()) <= (1e-5 if dt == "f32" else TOL[dt]), k
    mb.ffi.default_handle(0).check_status()
