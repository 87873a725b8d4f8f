"""What a context hands to the native call sequences (CPU, with a stand-in for the device state)."""

import types

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
