"""Host side of the engines (mamba_rs_b200/model.py) that needs no GPU: what a call refuses before anything is
launched, devices by name, and which sequences of launches an engine keeps recorded."""
import gc

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


def test_a_step_refuses_more_sequences_than_the_state_holds():
    bb = mb.GpuMambaBackbone(weights(), 2)
    with pytest.raises(ValueError, match="holds 2"):
        bb.step(torch.zeros(3, 16))


def test_calls_refuse_rows_on_another_device():
    bb = mb.GpuMambaBackbone(weights(), 2)
    with pytest.raises(TypeError, match="device|meta"):
        bb.step(torch.zeros(2, 16, device="meta"))


@pytest.mark.parametrize("device", ["cpu", torch.device("cpu")])
def test_weights_take_a_device_by_name(device):
    w = weights(device).init_random(1)
    assert w.device == w.master.device == torch.device("cpu") and bool(w.master.abs().sum() > 0)
    assert mb.MambaLMTrainer(w)._plans == {}


class FakeGraph:
    made = 0

    def __init__(self, launch):
        FakeGraph.made += 1
        self.launch = launch

    def replay(self):
        self.launch()


@pytest.fixture
def shelf(monkeypatch):
    s = model._Shelf(torch.device("cpu"), limit=100)
    monkeypatch.setattr(s, "record", lambda launch: (FakeGraph(launch), launch))
    monkeypatch.setattr(model.ops, "_on", lambda dev: __import__("contextlib").nullcontext())
    FakeGraph.made = 0
    return s


def test_a_sequence_is_recorded_when_it_comes_for_the_third_time(shelf):
    r, ran = model._Replay(shelf, 10), []
    for i in range(6):
        r.run("a", lambda: ran.append(i))
        assert (FakeGraph.made, len(ran)) == (int(i >= 2), i + 1)


def test_buffers_in_rotation_do_not_record_on_every_call(shelf):
    """More addresses than are kept: as many as there is room for are replayed, the others launched."""
    r, n, ran = model._Replay(shelf, 1), shelf.KEEP + 4, []
    for i in range(30 * n):
        r.run(i % n, lambda: ran.append(0))
    assert FakeGraph.made == shelf.KEEP == len(r.kept) and len(ran) == 30 * n


def test_one_limit_holds_over_all_plans_and_idle_recordings_give_way(shelf):
    a, b, big = model._Replay(shelf, 60), model._Replay(shelf, 50), model._Replay(shelf, 101)
    for r in (a, big, b):
        for _ in range(5):
            r.run("x", lambda: None)
    assert list(a.kept) == ["x"] and not b.kept and not big.kept  # 60 + 50 > 100; a is in use
    for _ in range(shelf.PATIENCE):
        b.run("x", lambda: None)
    assert not a.kept and not a.seen and list(b.kept) == ["x"] and sum(p.nbytes for p in shelf.places) == 50
    a.run("x", lambda: None)
    assert not a.kept  # and is counted from the start again


def test_what_a_dropped_plan_kept_makes_room(shelf):
    a = model._Replay(shelf, 60)
    for _ in range(3):
        a.run("x", lambda: None)
    assert len(shelf.places) == 1
    del a
    gc.collect()
    assert not shelf.places


def test_a_sequence_that_cannot_be_recorded_is_launched(shelf, monkeypatch):
    monkeypatch.setattr(shelf, "record", lambda launch: None)
    r, ran = model._Replay(shelf, 10), []
    for _ in range(4):
        r.run("a", lambda: ran.append(0))
    assert len(ran) == 4 and not r.kept and not shelf.places


def test_an_engine_goes_without_the_cycle_collector():
    import weakref
    bb = mb.GpuMambaBackbone(weights(), 2)
    bb._prefill_plan(2, 3) if torch.cuda.is_available() else None
    ref = weakref.ref(bb._shelf)
    gc.disable()
    try:
        del bb
        assert ref() is None
    finally:
        gc.enable()
