"""GPU parity tests of the Mamba-3 SISO SSD forward against the CPU oracle's
sequential definition.  Tolerances as for Mamba-1: 1e-4 (f32 storage), 2e-2
(bf16 / f16 storage), max-abs relative to the max-abs reference."""
import numpy as np
import pytest

import oracle
from helpers import TOL, rel_err, to_dev, torch_dtype
from mamba_rs_b200 import synth

pytestmark = pytest.mark.gpu
ARGS = ("x", "K", "Q", "dt", "trap", "adt", "Dh")


def rounded(i, dt):
    return {k: (synth.round_to(v, dt) if k in ("x", "K", "Q") else v) for k, v in i.items()}


def run_gpu(i, dt, dev, **kw):
    import torch

    import mamba_rs_b200 as mb
    td = torch_dtype(dt)
    B, T, nh, N = i["K"].shape
    hd = i["x"].shape[2] // nh
    ssm = torch.zeros(B, nh, hd, N, device=dev)
    ks = torch.zeros(B, nh, N, device=dev)
    vs = torch.zeros(B, nh, hd, device=dev)
    y = mb.m3_ssd_fwd(to_dev(i["x"], dev, td), to_dev(i["K"], dev, td), to_dev(i["Q"], dev, td),
                      to_dev(i["dt"], dev), to_dev(i["trap"], dev), to_dev(i["adt"], dev), to_dev(i["Dh"], dev),
                      ssm_state=ssm, k_state=ks, v_state=vs, **kw)
    torch.cuda.synchronize()
    mb.ffi.default_handle(0).check_status()
    return y.float().cpu().numpy(), ssm.cpu().numpy(), ks.cpu().numpy(), vs.cpu().numpy()


# shapes of the reference's own unit parity test (tests/m3_chunked_fwd_unit_parity.rs:20-31:
# B=2,T=10,nh=2,hd=4,ds=4), its limits (hd 32, N 64), and beyond them
SEQ_SHAPES = [(2, 10, 2, 4, 4), (1, 64, 3, 16, 16), (2, 100, 2, 32, 64), (1, 70, 2, 64, 128), (1, 33, 1, 8, 24)]


@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("shape", SEQ_SHAPES, ids=lambda s: "B%dT%dnh%dhd%dN%d" % s)
def test_sequential_kernel_matches_oracle(cuda_dev, shape, dt):
    B, T, nh, hd, N = shape
    i = rounded(synth.m3_ssd_inputs(B, T, nh, hd, N, seed=T), dt)
    ref = oracle.m3_ssd_fwd(*[i[k] for k in ARGS])
    y, ssm, ks, vs = run_gpu(i, dt, cuda_dev, force_sequential=True)
    assert rel_err(y, ref["y"]) <= TOL[dt]
    assert rel_err(ssm, ref["ssm_state"]) <= 1e-4
    np.testing.assert_array_equal(ks, ref["k_state"])
    np.testing.assert_array_equal(vs, ref["v_state"])


def test_sequential_kernel_carries_state(cuda_dev):
    import torch

    import mamba_rs_b200 as mb
    i = synth.m3_ssd_inputs(1, 60, 2, 16, 32, seed=5)
    whole = oracle.m3_ssd_fwd(*[i[k] for k in ARGS])
    dev = cuda_dev
    ssm = torch.zeros(1, 2, 16, 32, device=dev)
    ks = torch.zeros(1, 2, 32, device=dev)
    vs = torch.zeros(1, 2, 16, device=dev)
    ys = []
    for lo, hi, carry in ((0, 25, False), (25, 60, True)):
        sl = {k: (np.ascontiguousarray(i[k][:, lo:hi]) if k != "Dh" else i[k]) for k in ARGS}
        ys.append(mb.m3_ssd_fwd(*[to_dev(sl[k], dev) for k in ARGS], ssm_state=ssm, k_state=ks, v_state=vs,
                                carry_in=carry))
    torch.cuda.synchronize()
    assert rel_err(torch.cat(ys, 1).cpu().numpy(), whole["y"]) <= 1e-5
    assert rel_err(ssm.cpu().numpy(), whole["ssm_state"]) <= 1e-5


# tensor-core path: hd = 64, N = 128, 16-bit storage; T around the 128-step chunk
TC_SHAPES = [(1, 128, 1), (2, 256, 2), (1, 1, 1), (1, 100, 2), (1, 129, 1), (2, 300, 3), (1, 1000, 2)]


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("shape", TC_SHAPES, ids=lambda s: "B%dT%dnh%d" % s)
def test_tensor_core_kernel_matches_oracle(cuda_dev, shape, dt):
    B, T, nh = shape
    i = rounded(synth.m3_ssd_inputs(B, T, nh, 64, 128, seed=T + 1), dt)
    ref = oracle.m3_ssd_fwd(*[i[k] for k in ARGS])
    y, ssm, ks, vs = run_gpu(i, dt, cuda_dev)
    assert rel_err(y, ref["y"]) <= TOL[dt]
    assert rel_err(ssm, ref["ssm_state"]) <= TOL[dt]  # 16-bit operands feed the state GEMM
    np.testing.assert_array_equal(ks, ref["k_state"])
    np.testing.assert_array_equal(vs, ref["v_state"])


# the reference's own limits (headdim 32, d_state 64) and other multiples of 8: the
# kernel pads its tiles to 64 / 128 columns with zeros
PADDED_SHAPES = [(2, 200, 2, 32, 64), (1, 130, 3, 8, 8), (1, 300, 2, 24, 40), (1, 129, 1, 64, 16), (1, 64, 2, 16, 128)]


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("shape", PADDED_SHAPES, ids=lambda s: "B%dT%dnh%dhd%dN%d" % s)
def test_tensor_core_kernel_with_padded_head_and_state_dims(cuda_dev, shape, dt):
    B, T, nh, hd, N = shape
    i = rounded(synth.m3_ssd_inputs(B, T, nh, hd, N, seed=T + hd), dt)
    ref = oracle.m3_ssd_fwd(*[i[k] for k in ARGS])
    y, ssm, ks, vs = run_gpu(i, dt, cuda_dev)
    assert rel_err(y, ref["y"]) <= TOL[dt]
    assert rel_err(ssm, ref["ssm_state"]) <= TOL[dt]
    np.testing.assert_array_equal(ks, ref["k_state"])
    np.testing.assert_array_equal(vs, ref["v_state"])
    y2, ssm2, _, _ = run_gpu(i, dt, cuda_dev, force_sequential=True)
    assert rel_err(y, y2) <= TOL[dt]


def test_tensor_core_and_sequential_kernels_agree(cuda_dev):
    i = rounded(synth.m3_ssd_inputs(2, 520, 4, 64, 128, seed=9), "bf16")
    y1, s1, _, _ = run_gpu(i, "bf16", cuda_dev)
    y2, s2, _, _ = run_gpu(i, "bf16", cuda_dev, force_sequential=True)
    assert rel_err(y1, y2) <= TOL["bf16"]
    assert rel_err(s1, s2) <= TOL["bf16"]


def test_tensor_core_kernel_at_config4_size_agrees_with_sequential_and_is_linear_in_x(cuda_dev):
    """Benchmark geometry (B 8, L 4096, 32 heads x 64, d_state 128, bf16): the
    tcgen05 kernel against the sequential kernel on the same device tensors, and
    the size-independent property y(x1 + x2) = y(x1) + y(x2) - y(0) with y(0) = 0."""
    import torch

    import mamba_rs_b200 as mb
    B, T, nh, hd, N = 8, 4096, 32, 64, 128
    g = torch.Generator(device="cpu").manual_seed(4)
    bf = torch.bfloat16
    dev = cuda_dev
    x1 = torch.randn(B, T, nh * hd, generator=g).to(dev).to(bf)
    x2 = torch.randn(B, T, nh * hd, generator=g).to(dev).to(bf)
    K = (torch.randn(B, T, nh, N, generator=g) * N ** -0.25).to(dev).to(bf)
    Q = (torch.randn(B, T, nh, N, generator=g) * N ** -0.25).to(dev).to(bf)
    A = -torch.exp(torch.rand(nh, generator=g) * np.log(16.0))
    dt = torch.nn.functional.softplus(0.5 * torch.randn(B, T, nh, generator=g) - 4.0)
    trap = torch.sigmoid(torch.randn(B, T, nh, generator=g))
    adt = (A * dt).to(dev).contiguous()
    dt, trap = dt.to(dev).contiguous(), trap.to(dev).contiguous()
    Dh = torch.ones(nh, device=dev)
    s_tc = torch.zeros(B, nh, hd, N, device=dev)
    s_seq = torch.zeros(B, nh, hd, N, device=dev)
    y_tc = mb.m3_ssd_fwd(x1, K, Q, dt, trap, adt, Dh, ssm_state=s_tc).float()
    y_seq = mb.m3_ssd_fwd(x1, K, Q, dt, trap, adt, Dh, ssm_state=s_seq, force_sequential=True).float()
    torch.cuda.synchronize()
    mb.ffi.default_handle(0).check_status()
    den = y_seq.abs().max()
    assert float((y_tc - y_seq).abs().max() / den) <= TOL["bf16"]
    assert float((s_tc - s_seq).abs().max() / s_seq.abs().max()) <= TOL["bf16"]
    del y_seq
    x12 = (x1.float() + x2.float()).to(bf)  # rounding of the sum stays inside the tolerance
    y2 = mb.m3_ssd_fwd(x2, K, Q, dt, trap, adt, Dh).float()
    y12 = mb.m3_ssd_fwd(x12, K, Q, dt, trap, adt, Dh).float()
    torch.cuda.synchronize()
    assert float((y12 - (y_tc + y2)).abs().max() / y12.abs().max()) <= TOL["bf16"]


# a stream in windows: the tensor-core kernel from a carried state (windows beyond the short ones the
# sequential kernel keeps), ragged windows around the 128-step chunk, padded head / state sizes, and a
# head count that is no multiple of 4; state held to the f32 bar because the carried form splits every
# rounded operand in two
CARRY_SHAPES = [((25, 1, 40), 1, 2, 64, 128), ((128, 256, 3), 2, 4, 64, 128), ((1, 129, 300), 1, 3, 64, 128),
                ((60, 70), 2, 2, 32, 64), ((30, 127, 128), 1, 2, 24, 40), ((200, 1, 1), 1, 40, 72, 96)]


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("shape", CARRY_SHAPES, ids=lambda s: "T%s_B%dnh%dhd%dN%d" % ("_".join(map(str, s[0])), *s[1:]))
def test_windows_of_a_stream_carry_state(cuda_dev, shape, dt):
    import torch

    import mamba_rs_b200 as mb
    cuts, B, nh, hd, N = shape
    i = rounded(synth.m3_ssd_inputs(B, sum(cuts), nh, hd, N, seed=sum(cuts)), dt)
    whole = oracle.m3_ssd_fwd(*[i[k] for k in ARGS])
    td = torch_dtype(dt)
    ssm, ks, vs = (torch.zeros(*s, device=cuda_dev) for s in ((B, nh, hd, N), (B, nh, N), (B, nh, hd)))
    ys, lo = [], 0
    for n in cuts:
        sl = {k: (np.ascontiguousarray(i[k][:, lo:lo + n]) if k != "Dh" else i[k]) for k in ARGS}
        ys.append(mb.m3_ssd_fwd(*[to_dev(sl[k], cuda_dev, td if k in ("x", "K", "Q") else None) for k in ARGS],
                                ssm_state=ssm, k_state=ks, v_state=vs, carry_in=True))
        lo += n
    torch.cuda.synchronize()
    mb.ffi.default_handle(0).check_status()
    assert rel_err(torch.cat(ys, 1).float().cpu().numpy(), whole["y"]) <= TOL[dt]
    assert rel_err(ssm.cpu().numpy(), whole["ssm_state"]) <= 1e-4
    np.testing.assert_array_equal(ks.cpu().numpy(), whole["k_state"])
    np.testing.assert_array_equal(vs.cpu().numpy(), whole["v_state"])


# few (sample, head) pairs: the chunks are divided over the CTAs of a cluster; fewer chunks than ranks, ranks
# left without chunks, a last chunk of one step
CLUSTER_SHAPES = [(1, 257, 1, 64, 128), (1, 640, 3, 64, 128), (2, 1153, 2, 32, 64), (1, 1290, 4, 64, 128),
                  (2, 2048, 37, 64, 128)]


@pytest.mark.parametrize("carry", [False, True])
@pytest.mark.parametrize("shape", CLUSTER_SHAPES, ids=lambda s: "B%dT%dnh%dhd%dN%d" % s)
def test_chunks_divided_over_a_cluster_match_sequential(cuda_dev, shape, carry):
    import torch

    import mamba_rs_b200 as mb
    i = rounded(synth.m3_ssd_inputs(*shape, seed=shape[1]), "bf16")
    B, T, nh, hd, N = shape
    g = torch.Generator().manual_seed(T)
    st0 = [torch.randn(*s, generator=g).to(cuda_dev) for s in ((B, nh, hd, N), (B, nh, N), (B, nh, hd))]
    args = [to_dev(i[k], cuda_dev, torch.bfloat16 if k in ("x", "K", "Q") else None) for k in ARGS]
    out = []
    for seq in (False, True):
        ssm, ks, vs = (t.clone() for t in st0)
        y = mb.m3_ssd_fwd(*args, ssm_state=ssm, k_state=ks, v_state=vs, carry_in=carry, force_sequential=seq)
        out.append([t.float().cpu().numpy() for t in (y, ssm, ks, vs)])
    mb.ffi.default_handle(0).check_status()
    assert rel_err(out[0][0], out[1][0]) <= TOL["bf16"]
    assert rel_err(out[0][1], out[1][1]) <= (1e-4 if carry else TOL["bf16"])
    np.testing.assert_array_equal(out[0][2], out[1][2])
    np.testing.assert_array_equal(out[0][3], out[1][3])


@pytest.mark.parametrize("T,nh", [(7169, 1), (7177, 3)])
def test_a_divided_window_starts_from_the_state_that_entered(cuda_dev, T, nh):
    """57 chunks over eight CTAs: the last has one short chunk and then replaces the state in place, while the
    first still has eight to walk in full from the one that entered.  Every call must be the same."""
    import torch

    import mamba_rs_b200 as mb
    i = rounded(synth.m3_ssd_inputs(1, T, nh, 64, 128, seed=T), "bf16")
    args = [to_dev(i[k], cuda_dev, torch.bfloat16 if k in ("x", "K", "Q") else None) for k in ARGS]
    g = torch.Generator().manual_seed(T)
    st0 = [100 * torch.randn(*s, generator=g).to(cuda_dev) for s in ((1, nh, 64, 128), (1, nh, 128), (1, nh, 64))]

    def call(seq):
        ssm, ks, vs = (t.clone() for t in st0)
        y = mb.m3_ssd_fwd(*args, ssm_state=ssm, k_state=ks, v_state=vs, carry_in=True, force_sequential=seq)
        return y, ssm
    y, ssm = call(False)
    ry, rs = call(True)
    # the state that entered fills the first rows of y (100 against the inputs' 1), so a wrong one shows there
    assert rel_err(y.float().cpu().numpy(), ry.float().cpu().numpy()) <= TOL["bf16"]
    assert rel_err(ssm.cpu().numpy(), rs.cpu().numpy()) <= 1e-4
    for _ in range(20):
        y2, ssm2 = call(False)
        assert torch.equal(y2, y) and torch.equal(ssm2, ssm)
    mb.ffi.default_handle(0).check_status()


def window_f64(i, st):
    """The sequential definition in 64 bits: y [B,T,nh*hd] and the state after the window."""
    B, T, nh, N = i["K"].shape
    h, kp, vp = (s.astype(np.float64) for s in st)
    d = {k: i[k].astype(np.float64) for k in ARGS}
    y = np.empty((B, T, nh, h.shape[2]))
    for t in range(T):
        al, v = np.exp(d["adt"][:, t]), d["x"][:, t].reshape(B, nh, -1)
        be, ga = al * d["dt"][:, t] * (1 - d["trap"][:, t]), d["trap"][:, t] * d["dt"][:, t]
        h = al[..., None, None] * h + (be[..., None] * vp)[..., None] * kp[:, :, None] + (ga[..., None] * v)[..., None] * d["K"][:, t][:, :, None]
        y[:, t] = np.einsum("bhpn,bhn->bhp", h, d["Q"][:, t]) + d["Dh"][:, None] * v
        kp, vp = d["K"][:, t], v
    return y.reshape(B, T, -1), h


# (dtype, T, factor on x and the state, factor on K and Q): the divided form, one CTA a head, and what f16 cannot
# hold as products (65504) or remainders (6e-8)
@pytest.mark.parametrize("dt,T,nh,fx,fk", [("bf16", 1000, 4, 1, 1), ("bf16", 200, 160, 1, 1), ("bf16", 300, 2, 1e-3, 1),
                                           ("f16", 1000, 4, 1, 1), ("f16", 300, 2, 1e-3, 1), ("f16", 300, 2, 1, 1e-2),
                                           ("f16", 300, 2, 1e-2, 200)])
def test_a_carried_window_is_as_exact_as_the_sequential_definition(cuda_dev, dt, T, nh, fx, fk):
    import torch

    import mamba_rs_b200 as mb
    hd, N = 64, 128
    i = synth.m3_ssd_inputs(1, T, nh, hd, N, seed=T)
    i["Dh"] = 0 * i["Dh"]  # (the skip would hide the scan's part of y)
    i["x"], i["K"], i["Q"] = i["x"] * np.float32(fx), i["K"] * np.float32(fk), i["Q"] * np.float32(fk)
    i = rounded(i, dt)
    rng = np.random.default_rng(T)
    st0 = [(f * rng.standard_normal(s)).astype(np.float32) for f, s in ((fx * fk, (1, nh, hd, N)), (fk, (1, nh, N)), (fx, (1, nh, hd)))]
    ref = window_f64(i, st0)
    args = [to_dev(i[k], cuda_dev, torch_dtype(dt) if k in ("x", "K", "Q") else None) for k in ARGS]
    err = []
    for seq in (False, True):
        ssm, ks, vs = (to_dev(s, cuda_dev) for s in st0)
        y = mb.m3_ssd_fwd(*args, ssm_state=ssm, k_state=ks, v_state=vs, carry_in=True, force_sequential=seq)
        err.append([np.linalg.norm(a.double().cpu().numpy() - r) / np.linalg.norm(r) for a, r in zip((y, ssm), ref)])
    mb.ffi.default_handle(0).check_status()
    # y: both are the rounding of the store; state: f32 sums in another order, a few 2^-24 of 128 terms a chunk
    assert err[0][0] <= 1.01 * err[1][0], err
    assert err[0][1] <= max(err[1][1], 2e-6), err


@pytest.mark.parametrize("N", [8, 40, 96, 100])
def test_an_infinite_input_stays_infinite_beside_the_states_that_are_not_there(cuda_dev, N):
    """The lanes past d_state hold zeros; an infinite x must not make a NaN of them and carry it into y."""
    i = synth.m3_ssd_inputs(1, 12, 1, 16, N, seed=N)
    for k in ("K", "Q"):
        i[k] = np.abs(i[k]) + np.float32(0.1)
    i["Dh"], i["x"][0, 5, 3] = np.abs(i["Dh"]), np.inf
    y, ssm, _, _ = run_gpu(i, "f32", cuda_dev, force_sequential=True)
    assert np.isinf(y[0, 5:, 3]).all() and np.isfinite(np.delete(y, 3, axis=2)).all()
    assert np.isinf(ssm[0, 0, 3]).all()


# More (sample, head) pairs than SMs run two CTAs per SM, fewer one: the same arithmetic in the same order, so a batch
# of 150 or more pairs must give, bit for bit, what its first and its last samples give in calls of fewer than 148.  Of a
# carried window y's sums are in another order there: f32 sums of up to 500 terms differ by less than 1e-5 of the
# largest value, and then by one rounding to the storage type at most.
@pytest.mark.parametrize("dt", ["bf16", "f16", "carried"])
@pytest.mark.parametrize("case", [(10, 1, 16, 64, 128), (10, 127, 15, 32, 64), (10, 128, 16, 8, 16), (10, 129, 15, 64, 128),
                                  (10, 300, 16, 64, 72), (10, 513, 16, 56, 128)], ids=lambda c: "B%dT%dnh%dhd%dN%d" % c)
def test_two_ctas_per_sm_give_the_same_bits(cuda_dev, case, dt):
    import torch

    import mamba_rs_b200 as mb
    B, T, nh, hd, N = case
    carried = dt == "carried"
    td = torch.float16 if dt == "f16" else torch.bfloat16
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    rn = lambda *s: torch.randn(*s, device=cuda_dev, generator=g)  # noqa: E731
    x, K, Q = rn(B, T, nh * hd).to(td), (0.3 * rn(B, T, nh, N)).to(td), (0.3 * rn(B, T, nh, N)).to(td)
    dt_, trap = torch.nn.functional.softplus(rn(B, T, nh) - 2), torch.sigmoid(rn(B, T, nh))
    adt, Dh = -dt_ * torch.rand(nh, device=cuda_dev, generator=g) * 4, rn(nh)
    h0, k0, v0 = rn(B, nh, hd, N), 0.3 * rn(B, nh, N), rn(B, nh, hd)

    def call(lo, hi):
        c = lambda t: t[lo:hi].contiguous()  # noqa: E731
        new = lambda t: t[lo:hi].clone() if carried else torch.full_like(t[lo:hi], float("nan"))  # noqa: E731
        st = dict(ssm_state=new(h0), k_state=new(k0), v_state=new(v0))
        y = mb.m3_ssd_fwd(c(x), c(K), c(Q), c(dt_), c(trap), c(adt), Dh, carry_in=carried, **st)
        return [y, st["ssm_state"], st["k_state"], st["v_state"]]

    whole = call(0, B)
    for lo, hi in ((0, B - 1), (1, B)):
        for i, (a, b) in enumerate(zip(whole, call(lo, hi))):
            assert torch.isfinite(a.float()).all()
            if carried and i == 0:
                a, b = a[lo:hi].float(), b.float()
                assert bool(((a - b).abs() <= b.abs() / 128 + 1e-5 * b.abs().max()).all())
            else:
                assert torch.equal(a[lo:hi], b)
    mb.ffi.default_handle(0).check_status()


# Pairs that two CTAs per SM take are not divided over clusters, however long: the state has the bits that nine tenths
# of the batch, which are undivided pairs of one CTA, give in a call of their own.
@pytest.mark.parametrize("case", [(10, 4096, 15, True), (10, 16384, 15, False)], ids=lambda c: "B%dT%dnh%dcarry%d" % c)
def test_more_pairs_than_sms_are_not_divided(cuda_dev, case):
    import torch

    import mamba_rs_b200 as mb
    (B, T, nh, carried), hd, N = case, 64, 128
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    rn = lambda *s: torch.randn(*s, device=cuda_dev, generator=g)  # noqa: E731
    x, K, Q = [rn(B, T, nh, n).mul_(0.3).to(torch.bfloat16).view(B, T, -1) for n in (hd, N, N)]
    dt_, trap = torch.nn.functional.softplus(rn(B, T, nh) - 2), torch.sigmoid(rn(B, T, nh))
    adt, Dh = -dt_ * 0.01, rn(nh)  # slow enough for every chunk's roundings to reach the end
    h0, k0, v0 = rn(B, nh, hd, N), 0.3 * rn(B, nh, N), rn(B, nh, hd)

    def call(n):
        st = dict(ssm_state=h0[:n].clone(), k_state=k0[:n].clone(), v_state=v0[:n].clone())
        mb.m3_ssd_fwd(x[:n], K[:n].view(n, T, nh, N), Q[:n].view(n, T, nh, N), dt_[:n], trap[:n], adt[:n], Dh, carry_in=carried, **st)
        return st["ssm_state"]

    assert torch.equal(call(B)[:9], call(9))
    mb.ffi.default_handle(0).check_status()


# A short carried window keeps an infinite input to its own step, row and what follows, also where two CTAs per SM would
# be faster: the chunk's masked products would bring 0 * infinity to every step of the row.
@pytest.mark.parametrize("T", [16, 20])
def test_a_short_carried_window_keeps_an_infinite_input_to_its_row(cuda_dev, T):
    import torch

    import mamba_rs_b200 as mb
    B, nh, hd, N, at = 8, 32, 64, 128, T - 4
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    rn = lambda *s: torch.randn(*s, device=cuda_dev, generator=g)  # noqa: E731
    x, K, Q = [rn(B, T, nh, n).mul_(0.3).to(torch.bfloat16) for n in (hd, N, N)]
    x[3, at, 7, 21] = float("inf")
    dt_, trap = torch.nn.functional.softplus(rn(B, T, nh) - 2), torch.sigmoid(rn(B, T, nh))
    st = dict(ssm_state=rn(B, nh, hd, N), k_state=0.3 * rn(B, nh, N), v_state=rn(B, nh, hd))
    y = mb.m3_ssd_fwd(x.view(B, T, -1), K, Q, dt_, trap, -dt_, rn(nh), carry_in=True, **st).view(B, T, nh, hd)
    finite = torch.ones_like(y, dtype=torch.bool)
    finite[3, at:, 7, 21] = False
    assert torch.equal(torch.isfinite(y), finite) and bool(torch.isinf(st["ssm_state"][3, 7, 21]).all())
    mb.ffi.default_handle(0).check_status()
