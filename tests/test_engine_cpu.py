"""Host side of the engines (mamba_rs_b200/model.py) that needs no GPU: what a call refuses before anything is
launched, and devices by name."""
import pytest
import torch

import mamba_rs_b200 as mb
from mamba_rs_b200 import model


def weights(device="cpu"):
    return mb.MambaWeights(mb.MambaConfig(d_model=16, n_layers=1), device, dtype=torch.float32, vocab=8)


@pytest.mark.parametrize("width", [8, 24])
def test_a_step_refuses_rows_of_another_width(width):
    """(The one-launch kernel would read and write d_model values of every row whatever its length.)"""
    bb = mb.GpuMambaBackbone(weights(), 2)
    with pytest.raises(TypeError, match="16"):
        bb.step(torch.zeros(2, width))


def test_calls_refuse_rows_on_another_device():
    bb = mb.GpuMambaBackbone(weights(), 2)
    with pytest.raises(TypeError, match="device|meta"):
        bb.step(torch.zeros(2, 16, device="meta"))


@pytest.mark.parametrize("device", ["cpu", torch.device("cpu")])
def test_weights_take_a_device_by_name(device):
    w = weights(device).init_random(1)
    assert w.device == w.master.device == torch.device("cpu") and bool(w.master.abs().sum() > 0)
    assert mb.MambaLMTrainer(w)._plans == {}
