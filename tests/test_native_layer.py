"""What a context hands to the native call sequences, and the counters that they share (CPU, with a stand-in for the device state)."""

import types

import pytest
import torch

from dist_moe_b200 import _native, _runtime


def test_the_barrier_timeout_is_the_one_of_the_call(monkeypatch):
    buffer = types.SimpleNamespace(local=lambda: torch.zeros(16), peer_ptrs=torch.zeros(1), peer_pads=torch.zeros(1))
    config = types.SimpleNamespace(max_num_local_input_tokens=4, hidden_dim=8, intermediate_dim=8, top_k=2, num_experts=2,
                                   activation="swiglu", swiglu_alpha=1.0, swiglu_limit=7.0, block_scaled=None)
    one = torch.zeros(1)
    state = types.SimpleNamespace(config=config, arena=one, dispatch=buffer, combine=buffer, routing=buffer, saved_bytes=one,
                                  buffer_offsets=one, peak_min_free=one, slot_selector=one, moe_layer_id=one,
                                  route_workspace=one, gather_flags=one, status=one, route_workspace_words=1, slot_bytes=128,
                                  capacity_rows=4, rank=0, ep=2, e_local=1, num_slots=1, num_sms=0)

    def timeout():
        return _runtime.ContextState.native_layer(state)._obj.barrier_timeout_ns

    assert timeout() == _runtime.BARRIER_TIMEOUT_NS
    monkeypatch.setattr(_runtime, "BARRIER_TIMEOUT_NS", 123)
    assert timeout() == 123
    assert isinstance(state._native_layer, _native.LayerContext)


# The counters of the fused dispatch, which no call clears in front of its launch, are clear again after a context's reset and after a
# reported failure.
def _state(code):
    one = lambda n=1: torch.zeros(n, dtype=torch.int64)  # noqa: E731
    state = types.SimpleNamespace(
        num_slots=1, slot_bytes=128, arena_bytes=1024, reserved_scratch_bytes=0, buffer_offsets=one(2), saved_bytes=one(),
        peak_min_free=one(2), moe_layer_id=one(), device=torch.device("cpu"),
        status=torch.tensor([code, 3, 2, 1, 0, 0, 0, 0], dtype=torch.int32), gather_flags=torch.full((9,), 5, dtype=torch.int32))
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
