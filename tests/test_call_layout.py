"""What a call keeps on its context is its layout alone, by kind; the device guard is free only on the current device (CPU)."""

import types

import pytest
import torch

from dist_moe_b200 import _bf16, _blockscaled, _call


def test_layouts_follow_the_kind_of_the_call():
    state = types.SimpleNamespace(e_local=6, ep=2, capacity_rows=100_000, config=types.SimpleNamespace(top_k=2))
    make = {"bf16": lambda T: _bf16._Call(state, T), "scratch": lambda T: _bf16._Call(state, T, False),
            "mxfp8": lambda T: _blockscaled._PlannedCall(state, T, None, None)}
    want = {(kind, T): (c.fields, c.at, c.words, c.size) for kind in make for T in (1, 33, 64)
            for c in [make[kind](T)] if not delattr(state, "_call_layout")}
    assert len({v[2] for v in want.values()}) == len(want)
    for kind, T in list(want) + list(reversed(list(want))):  # whatever the call before was
        for _ in range(2):
            c = make[kind](T)
            assert (c.fields, c.at, c.words, c.size) == want[kind, T]
    for fields, at, words, _ in want.values():  # 16-byte aligned, in order, without overlap
        ends = [at[n] + f[1] * f[0].itemsize for n, f in fields.items()]
        starts = list(at.values())
        assert all(s % 16 == 0 for s in starts) and all(e <= s for e, s in zip(ends, starts[1:] + [8 * words]))


@pytest.mark.parametrize("current,index,free", [(0, 0, True), (1, 0, False), (0, None, False)])
def test_device_guard(monkeypatch, current, index, free):
    made = []
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: current, raising=False)
    monkeypatch.setattr(torch.cuda, "device", lambda d: made.append(d) or _call._NOTHING)
    device = torch.device("cuda") if index is None else torch.device("cuda", index)
    with _call.on_device(device):
        pass
    assert made == ([] if free else [device])
