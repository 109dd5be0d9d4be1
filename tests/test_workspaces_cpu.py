"""Workspace sizes, which are asked for without a device: one that was sized for the largest call of a program
serves its smaller ones."""
import ctypes

import pytest

from mamba_rs_b200 import ffi


@pytest.mark.parametrize("N", [8, 16, 64])
@pytest.mark.parametrize("D", [64, 640, 1536, 5120])
def test_a_scan_forward_workspace_for_a_larger_batch_or_length_is_large_enough(D, N):
    size = ffi.lib().mamba_b200_sscan_fwd_workspace_bytes
    for T in (64, 192, 256, 500, 1021, 4096):
        got = [size(B, T, D, N) for B in range(1, 40)]
        assert got == sorted(got), (T, got)
        assert size(3, T - 40, D, N) <= size(3, T, D, N)


def layout(dtype, B, T, D, N=16, z_mode=1, lent=None):
    """(states a lane by warp roles or 0, consumer warps, time segments) of such a call; lent: bytes, None what it asks for."""
    if lent is None:
        lent = ffi.lib().mamba_b200_sscan_fwd_workspace_bytes(B, T, D, N)
    out = (ctypes.c_int * 3)()
    assert ffi.lib().mamba_b200_sscan_fwd_layout(dtype, B, T, D, N, z_mode, lent, out) == 0
    return tuple(out)


@pytest.mark.parametrize("dtype", [ffi.F32, ffi.BF16])
@pytest.mark.parametrize("shape", [(1, 1021, 1536), (4, 512, 256), (2, 700, 640), (1, 4096, 1536)])
def test_a_workspace_that_is_too_small_to_cut_with_is_like_none(dtype, shape):
    assert layout(dtype, *shape)[2] > 1
    assert layout(dtype, *shape, lent=4096) == layout(dtype, *shape, lent=0)
