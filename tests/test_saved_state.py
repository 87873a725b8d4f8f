"""The state a BF16 training call saves, as the registered operators hand it out and as views of the call's one buffer (CPU)."""

import types

import pytest
import torch

from dist_moe_b200 import _bf16

STATE = types.SimpleNamespace(e_local=6, ep=2, capacity_rows=1000)
NAMES = ("counts", "bwd", "fwd", "sct", "per_rank", "recv_rows", "need", "fwd_state")


def _call(T, norm):
    c = _bf16._Call(STATE, T).allocate("cpu")
    c.buf.random_(generator=torch.Generator().manual_seed(T))
    c.rstd = torch.rand(T, 2) if norm else None
    return c


@pytest.mark.parametrize("T", [1, 33, 64])
@pytest.mark.parametrize("norm", [False, True])
def test_saved_tensors_are_the_call(T, norm):
    c = _call(T, norm)
    saved = c.saved()
    shapes = [(6,), (12 * T,), (12 * T,), (12 * T,), (2,), (1,), (1,), (6,), (T, 2) if norm else (0,)]  # the operators' own
    assert [tuple(t.shape) for t in saved] == shapes
    for name, t in zip(NAMES, saved):
        want = getattr(c, name)
        assert want.dtype == t.dtype and want.data_ptr() == t.data_ptr() and torch.equal(want, t)
    back = _bf16._Call.from_saved(STATE, [t.detach() for t in saved], T)
    assert back.buf.data_ptr() == c.buf.data_ptr() and torch.equal(back.buf, c.buf)
    assert (back.T, back.size, back.max_rows) == (c.T, c.size, c.max_rows) and (back.rstd is None) == (not norm)


def test_tensors_that_moved_are_not_taken_for_the_buffer():
    saved = _call(33, False).saved()
    assert _bf16._Call.from_saved(STATE, [t.clone() for t in saved], 33) is None
    for i in range(8):
        some = list(saved)
        some[i] = some[i].clone()
        assert _bf16._Call.from_saved(STATE, some, 33) is None
    assert _bf16._Call.from_saved(STATE, saved, 34) is None
