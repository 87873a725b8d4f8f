"""The counters of the fused dispatch, which no call clears in front of its launch, are clear again after a context's reset and after a
reported failure (CPU, with a stand-in for the device state)."""

import types

import pytest
import torch

from dist_moe_b200 import _runtime


def _state(code):
    one = lambda n=1: torch.zeros(n, dtype=torch.int64)  # noqa: E731
    state = types.SimpleNamespace(
        num_slots=1, slot_bytes=128, arena_bytes=1024, reserved_scratch_bytes=0, buffer_offsets=one(2), saved_bytes=one(),
        peak_min_free=one(2), moe_layer_id=one(), device=torch.device("cpu"),
        status=torch.tensor([code, 3, 2, 1, 0, 0, 0, 0], dtype=torch.int32), gather_flags=torch.full((9,), 5, dtype=torch.int32))
    if hasattr(_runtime.ContextState, "clear_gather_flags"):
        state.clear_gather_flags = types.MethodType(_runtime.ContextState.clear_gather_flags, state)
    return state


def test_reset_clears_the_counters():
    state = _state(0)
    _runtime.ContextState.reset(state)
    assert not state.gather_flags.any()


@pytest.mark.parametrize("code", [0, 4, 5])
def test_a_reported_failure_clears_the_counters(code, monkeypatch):
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    state = _state(code)
    if code == 0:
        _runtime.ContextState.check_status(state)
        assert state.gather_flags.all()  # nothing failed: nothing is touched
        return
    with pytest.raises(RuntimeError):
        _runtime.ContextState.check_status(state)
    assert not state.gather_flags.any() and not state.status.any()
