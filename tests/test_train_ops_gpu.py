"""GPU parity of the rows around the scan: fused residual + RMSNorm (forward and
backward), embedding gather, softmax cross-entropy and AdamW, against the numpy
restatements in oracle/ (which cite the reference kernels they follow).
Tolerances: 1e-4 of the reference's max-abs for f32 results, 2e-2 for 16-bit ones."""
import numpy as np
import pytest

import oracle
from helpers import TOL, rel_err, to_dev, torch_dtype
from mamba_rs_b200 import synth

pytestmark = pytest.mark.gpu


def host(t):
    return t.float().cpu().numpy()


@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("shape", [(7, 128), (64, 768), (33, 2560), (5, 100), (3, 1), (2, 8192)],
                         ids=lambda s: "rows%d_dim%d" % s)
def test_residual_rmsnorm_forward_and_backward(cuda_dev, shape, dt):
    import torch

    import mamba_rs_b200 as mb
    rows, dim = shape
    rng = np.random.default_rng(rows + dim)
    res0 = rng.standard_normal((rows, dim)).astype(np.float32)
    branch = synth.round_to(rng.standard_normal((rows, dim)).astype(np.float32), dt)
    scale = (1.0 + 0.1 * rng.standard_normal(dim)).astype(np.float32)
    dy = synth.round_to(rng.standard_normal((rows, dim)).astype(np.float32), dt)
    td = torch_dtype(dt)
    d = lambda a, t_=None: to_dev(a, cuda_dev, t_)
    res = d(res0)
    y, rms = mb.residual_rmsnorm_fwd(res, d(branch, td), d(scale), eps=1e-5)
    x_ref, y_ref, rms_ref = oracle.residual_rmsnorm_fwd(res0, branch, scale, 1e-5)
    assert rel_err(host(res), x_ref) <= 1e-6
    assert rel_err(host(rms), rms_ref) <= 1e-5
    assert rel_err(host(y), y_ref) <= TOL[dt]
    # plain RMSNorm (no branch) leaves the residual untouched
    res2 = d(res0)
    y2, _ = mb.residual_rmsnorm_fwd(res2, None, d(scale), out_dtype=td)
    np.testing.assert_array_equal(host(res2), res0)
    assert rel_err(host(y2), oracle.residual_rmsnorm_fwd(res0, None, scale)[1]) <= TOL[dt]
    # backward: += into both outputs
    g0 = rng.standard_normal((rows, dim)).astype(np.float32)
    ds0 = rng.standard_normal(dim).astype(np.float32)
    d_res, d_scale = d(g0), d(ds0)
    mb.residual_rmsnorm_bwd(d(dy, td), res, d(scale), rms, d_res, d_scale)
    torch.cuda.synchronize()
    dx_ref, dsc_ref = oracle.residual_rmsnorm_bwd(dy, host(res), scale, host(rms))
    assert rel_err(host(d_res) - g0, dx_ref) <= 1e-4
    assert rel_err(host(d_scale) - ds0, dsc_ref) <= 1e-4
    mb.ffi.default_handle(0).check_status()


@pytest.mark.parametrize("dt", ["f32", "bf16"])
def test_embedding_gather(cuda_dev, dt):
    import torch

    import mamba_rs_b200 as mb
    V, dim, rows = 1000, 772, 300
    rng = np.random.default_rng(1)
    table = synth.round_to(rng.standard_normal((V, dim)).astype(np.float32), dt)
    ids = rng.integers(0, V, rows).astype(np.int32)
    ids[5], ids[6] = -1, V  # out of range: zero rows
    out = mb.embedding_gather(to_dev(table, cuda_dev, torch_dtype(dt)), to_dev(ids, cuda_dev))
    torch.cuda.synchronize()
    ref = table[np.clip(ids, 0, V - 1)]
    ref[[5, 6]] = 0.0
    np.testing.assert_array_equal(host(out), ref)


@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("shape", [(9, 50280), (33, 1000), (4, 77), (2, 120000)], ids=lambda s: "rows%d_V%d" % s)
def test_softmax_cross_entropy(cuda_dev, shape, dt):
    import torch

    import mamba_rs_b200 as mb
    rows, V = shape
    rng = np.random.default_rng(V)
    logits = synth.round_to((3.0 * rng.standard_normal((rows, V))).astype(np.float32), dt)
    tg = rng.integers(0, V, rows).astype(np.int32)
    tg[0] = -1  # a row that does not count
    loss, dl = mb.softmax_xent(to_dev(logits, cuda_dev, torch_dtype(dt)), to_dev(tg, cuda_dev), grad_scale=0.5)
    only_loss, none = mb.softmax_xent(to_dev(logits, cuda_dev, torch_dtype(dt)), to_dev(tg, cuda_dev), want_grad=False)
    torch.cuda.synchronize()
    loss_ref, g_ref = oracle.softmax_xent(logits, tg, 0.5)
    assert none is None
    assert rel_err(host(loss), loss_ref) <= 1e-5
    assert rel_err(host(only_loss), loss_ref) <= 1e-5
    assert rel_err(host(dl), g_ref) <= TOL[dt]
    assert float(host(dl)[0].max()) == 0.0 and float(host(loss)[0]) == 0.0
    mb.ffi.default_handle(0).check_status()


@pytest.mark.parametrize("lp", [None, "bf16", "f16"])
def test_adamw_matches_the_reference_update_rule(cuda_dev, lp):
    import torch

    import mamba_rs_b200 as mb
    n = 100003
    rng = np.random.default_rng(2)
    p0, g = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    m0, v0 = (0.1 * rng.standard_normal(n)).astype(np.float32), rng.random(n).astype(np.float32)
    hp = dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, wd=0.1)
    p_ref, m_ref, v_ref, bc = oracle.adamw_step(p0, g, m0, v0, hp["lr"], hp["beta1"], hp["beta2"], hp["eps"], hp["wd"], 7)
    d = lambda a: to_dev(a, cuda_dev)
    p, m, v = d(p0), d(m0), d(v0)
    lp_t = None if lp is None else torch.empty(n, device=cuda_dev, dtype=torch_dtype(lp))
    mb.adamw_step(p, d(g), m, v, d(np.array(bc, np.float32)), lr=hp["lr"], beta1=hp["beta1"], beta2=hp["beta2"],
                  eps=hp["eps"], weight_decay=hp["wd"], param_lp=lp_t)
    torch.cuda.synchronize()
    assert rel_err(host(p), p_ref) <= 1e-6
    assert rel_err(host(m), m_ref) <= 1e-6
    assert rel_err(host(v), v_ref) <= 1e-6
    if lp is not None:
        np.testing.assert_array_equal(host(lp_t), synth.round_to(host(p), lp))


@pytest.mark.parametrize("op", [0, 1, 2])
@pytest.mark.parametrize("size", [(1, 1, 1), (32, 64, 600), (33, 65, 33), (5, 100, 37), (64, 63, 1536), (31, 80, 520), (32, 768, 2050)],
                         ids=lambda s: "m%dn%dk%d" % s)
def test_sgemm_rows_matches_f64(cuda_dev, size, op):
    """Edges of the 32 x 64 tiles and of the parts of K, rows on and off 16 bytes, with and without a bias."""
    import torch

    from mamba_rs_b200 import ffi
    M, N, K = size
    h, lib = ffi.default_handle(0), ffi.lib()
    g = torch.Generator(device=cuda_dev).manual_seed(M + N + K)
    for pad in (0, 4, 3):
        new = lambda r, c: torch.randn(r, c + pad, device=cuda_dev, generator=g)[:, :c]  # noqa: E731
        a = new(K, M) if op == 2 else new(M, K)
        b = new(N, K) if op == 1 else new(K, N)
        c, bias = new(M, N), (torch.randn(N, device=cuda_dev, generator=g) if op != 2 and pad else None)
        ad, bd = a.double(), b.double()
        ref = ad @ bd if op == 0 else ad @ bd.t() if op == 1 else c.double() + ad.t() @ bd
        ref = ref if bias is None else ref + bias.double()
        rc = lib.mamba_b200_sgemm_rows(h.ptr, torch.cuda.current_stream().cuda_stream, op, a.data_ptr(), a.stride(0), b.data_ptr(),
                                       b.stride(0), None if bias is None else bias.data_ptr(), c.data_ptr(), c.stride(0), M, N, K)
        h.check(rc, "sgemm_rows")
        torch.cuda.synchronize()
        assert float((c.double() - ref).abs().max()) <= 3e-6 * K ** 0.5 * max(1.0, float(ref.abs().max()) / K ** 0.5)


@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("dim", [128, 132, 1024, 1028, 2048, 2052, 4096, 4100, 8192, 8196])
def test_residual_rmsnorm_forward_at_the_edges_of_its_kernels(cuda_dev, dim, dt):
    """Widths where the pieces of a thread or the threads of a row change, on both sides of few rows."""
    import torch

    import mamba_rs_b200 as mb
    td = torch_dtype(dt)
    g = torch.Generator(device=cuda_dev).manual_seed(dim)
    rn = lambda *s: torch.randn(*s, device=cuda_dev, generator=g)  # noqa: E731
    for rows in (1, 887, 888):
        res, br, sc = rn(rows, dim), rn(rows, dim).to(td), rn(dim)
        x = res.double() + br.double()
        rms = (x.square().mean(1) + 1e-5).sqrt()
        y, r = mb.residual_rmsnorm_fwd(res, br, sc)
        want = x / rms[:, None] * sc.double()
        assert float((res.double() - x).abs().max()) <= 1e-6 and float((r.double() / rms - 1).abs().max()) <= 1e-6
        assert float((y.double() - want).abs().max() / want.abs().max()) <= (1e-6 if dt == "f32" else 2 ** -8)


@pytest.mark.parametrize("op", [0, 1])
@pytest.mark.parametrize("size", [(32, 768, 50280), (12, 64, 50277), (33, 100, 4096), (32, 80, 1536)], ids=lambda s: "m%dn%dk%d" % s)
def test_sgemm_rows_stays_as_exact_over_a_long_contraction(cuda_dev, size, op):
    """One chain of f32 sums drifts by its length (1.4e-6 at 50280); chains of 256 whose sums are added up do
    not: about 2^-24 of the root of 256 steps each."""
    import torch

    from mamba_rs_b200 import ffi
    M, N, K = size
    h = ffi.default_handle(0)
    g = torch.Generator(device=cuda_dev).manual_seed(K)
    a = torch.randn(M, K, device=cuda_dev, generator=g)
    b = torch.randn(*((K, N) if op == 0 else (N, K)), device=cuda_dev, generator=g)
    bt, c = (b if op == 0 else b.t()), torch.empty(M, N, device=cuda_dev)
    rc = ffi.lib().mamba_b200_sgemm_rows(h.ptr, torch.cuda.current_stream().cuda_stream, op, a.data_ptr(), K, b.data_ptr(),
                                         b.stride(0), None, c.data_ptr(), N, M, N, K)
    h.check(rc, "sgemm_rows")
    ref = a.double() @ bt.double()
    assert float((c.double() - ref).norm() / ref.norm()) <= 4e-7


def test_sgemm_rows_gradient_takes_more_than_65535_tiles_of_rows(cuda_dev):
    import torch

    from mamba_rs_b200 import ffi
    M, N, K = 64 * 65536 + 1, 3, 2
    h = ffi.default_handle(0)
    g = torch.Generator(device=cuda_dev).manual_seed(1)
    a, b, c = (torch.randn(*s, device=cuda_dev, generator=g) for s in ((K, M), (K, N), (M, N)))
    ref = c.double() + a.double().t() @ b.double()
    rc = ffi.lib().mamba_b200_sgemm_rows(h.ptr, torch.cuda.current_stream().cuda_stream, 2, a.data_ptr(), M, b.data_ptr(), N, None,
                                         c.data_ptr(), N, M, N, K)
    h.check(rc, "sgemm_rows")
    assert float((c.double() - ref).abs().max()) <= 1e-5
