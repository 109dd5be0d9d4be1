"""Workspace sizes, which are asked for without a device: one that was sized for the largest call of a program
serves its smaller ones."""
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
