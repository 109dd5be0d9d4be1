"""Workspace sizes, which are asked for without a device: one that was sized for the largest call of a program
serves its smaller ones."""
import pytest

from helpers import scan_fwd_layout as layout
from mamba_rs_b200 import ffi


@pytest.mark.parametrize("N", [8, 16, 64])
@pytest.mark.parametrize("D", [64, 640, 1536, 5120])
def test_a_scan_forward_workspace_for_a_larger_batch_or_length_is_large_enough(D, N):
    size = ffi.lib().mamba_b200_sscan_fwd_workspace_bytes
    for T in (64, 192, 256, 500, 1021, 4096):
        got = [size(B, T, D, N) for B in range(1, 40)]
        assert got == sorted(got), (T, got)
        assert size(3, T - 40, D, N) <= size(3, T, D, N)


@pytest.mark.parametrize("dtype", [ffi.F32, ffi.BF16])
@pytest.mark.parametrize("shape", [(1, 1021, 1536), (4, 512, 256), (2, 700, 640), (1, 4096, 1536)])
def test_a_workspace_that_is_too_small_to_cut_with_is_like_none(dtype, shape):
    assert layout(dtype, *shape)[2] > 1
    assert layout(dtype, *shape, lent=4096) == layout(dtype, *shape, lent=0)


# Calls without a workspace on both sides of the line between the two kernels, by what was measured (us by the general
# kernel, by warp roles): steps past whole chunks, f32 without a gate, f32 with one, lengths that go on like the longer ones.
@pytest.mark.parametrize("case", [
    (ffi.BF16, 14, 37, 2416, 16, 1, False),   # 15.3, 19.8: 64 steps are walked
    (ffi.BF16, 9, 34, 1448, 16, 1, False),    # 8.3, 10.1
    (ffi.BF16, 8, 64, 1536, 16, 1, True),
    (ffi.F32, 25, 240, 1248, 16, 0, False),   # 51.3, 58.9: four CTAs of the general kernel an SM
    (ffi.F32, 10, 544, 3096, 16, 0, False),   # 110, 127
    (ffi.F32, 14, 1549, 1392, 16, 1, True),   # 254, 227
    (ffi.F32, 16, 2048, 1536, 16, 1, True),
    (ffi.BF16, 16, 2048, 1536, 16, 1, True),  # 363, 339
    (ffi.BF16, 16, 1504, 1536, 16, 1, True),
    (ffi.BF16, 16, 1065, 1544, 12, 1, True),  # 269, 185: B and C by plain loads
], ids=lambda c: "-".join(map(str, c)))
def test_the_scan_forward_takes_the_faster_kernel(case):
    *call, z_mode, roles = case
    assert (layout(*call, z_mode=z_mode, lent=0)[0] > 0) == roles
