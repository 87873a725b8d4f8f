"""A pass names its weights, ids and scores to the native sequences by address.  Whatever layout a tensor has at that moment, the
address is that of its elements in order, and another number of elements is refused (CPU: the sequences are replaced by a
recorder that reads the elements as the kernels would)."""

import contextlib
import ctypes
import types

import pytest
import torch

from dist_moe_b200 import _bf16, _blockscaled
from dist_moe_b200._execution import ExecutionOptions

E, F, D, T, K = 3, 4, 8, 5, 2


def _read(address, numel, dtype):
    raw = (ctypes.c_char * (numel * dtype.itemsize)).from_address(address)
    return torch.frombuffer(bytearray(raw.raw), dtype=dtype)


@pytest.fixture
def context(monkeypatch):
    """A stand-in for a context whose passes note the operands they are given."""
    seen = []

    def launch(fn, names, state, k, steps):
        seen.append(types.SimpleNamespace(
            w13=_read(k.w13, E * 2 * F * D, torch.bfloat16), w2=_read(k.w2, E * D * F, torch.bfloat16),
            ids=_read(k.ids, T * K, torch.int64), scores=_read(k.scores, T * K, torch.float32)))

    monkeypatch.setattr(_bf16, "launch", launch)
    monkeypatch.setattr(_blockscaled, "launch", launch)
    monkeypatch.setattr(_bf16, "on_device", lambda device: contextlib.nullcontext())
    config = types.SimpleNamespace(hidden_dim=D, intermediate_dim=F, top_k=K, num_experts=E, inference=False, wgrad_dtype=None)
    state = types.SimpleNamespace(config=config, e_local=E, ep=1, capacity_rows=1000, num_slots=1, num_layers_in_slot=1,
                                  device=torch.device("cpu"))
    return types.SimpleNamespace(config=config, _state=state, _closed=False, _context_id="none", seen=seen)


def _tensors():
    g = torch.Generator().manual_seed(3)
    x = torch.randn(T, D, generator=g).bfloat16()
    ids, scores = torch.randint(0, E, (T, K), generator=g), torch.rand(T, K, generator=g)
    w13, w2 = torch.randn(E, 2, F, D, generator=g).bfloat16(), torch.randn(E, D, F, generator=g).bfloat16()
    return x, ids, scores, w13, w2


def _apply(context, x, ids, scores, w13, w2):
    return _bf16._RegisteredBf16Function.apply(x, ids, scores, w13, w2, context, ExecutionOptions())


def _same(got, want):
    return torch.equal(got, want.reshape(-1))


def test_weights_whose_dimensions_merge_only_by_a_copy(context):
    """Gate and up projections stacked first, handed over as (E, 2, F, D): the entry point accepts them."""
    x, ids, scores, w13, w2 = _tensors()
    stacked = w13.transpose(0, 1).contiguous().transpose(0, 1).requires_grad_(True)
    assert not stacked.is_contiguous() and torch.equal(stacked, w13)
    out = _apply(context, x, ids, scores, stacked, w2)
    out.backward(torch.zeros_like(out))
    assert len(context.seen) > 1
    for k in context.seen:
        assert _same(k.w13, w13) and _same(k.w2, w2) and _same(k.ids, ids) and _same(k.scores, scores)


def _swapped(t):
    """The same values with the last two dimensions exchanged in memory."""
    return t.detach().transpose(-1, -2).contiguous().transpose(-1, -2)


@pytest.mark.parametrize("which", ["w13", "w2", "scores"])
def test_another_layout_between_forward_and_backward(context, which):
    x, ids, scores, w13, w2 = _tensors()
    leaves = {"w13": w13.requires_grad_(True), "w2": w2.requires_grad_(True), "scores": scores.requires_grad_(True)}
    out = _apply(context, x, ids, scores, w13, w2)
    want, forward = leaves[which].detach().clone(), len(context.seen)
    leaves[which].data = _swapped(leaves[which])
    assert not leaves[which].is_contiguous() and torch.equal(leaves[which], want)
    out.backward(torch.zeros_like(out))
    assert len(context.seen) > forward
    for k in context.seen:
        assert _same(getattr(k, which), want)


@pytest.mark.parametrize("which", ["w13", "w2", "scores"])
def test_another_size_between_forward_and_backward(context, which):
    x, ids, scores, w13, w2 = _tensors()
    leaves = {"w13": w13.requires_grad_(True), "w2": w2.requires_grad_(True), "scores": scores.requires_grad_(True)}
    out = _apply(context, x, ids, scores, w13, w2)
    forward = len(context.seen)
    leaves[which].data = leaves[which].detach()[:2].contiguous()
    with pytest.raises(RuntimeError):
        out.backward(torch.zeros_like(out))
    assert len(context.seen) == forward  # nothing was launched


def test_what_a_saved_tensor_hook_returns(context):
    x, ids, scores, w13, w2 = _tensors()
    w13.requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: _swapped(t) if t.ndim > 1 else t):
        out = _apply(context, x, ids, scores, w13, w2)
    out.backward(torch.zeros_like(out))
    for k in context.seen:
        assert _same(k.w13, w13.detach()) and _same(k.w2, w2) and _same(k.ids, ids) and _same(k.scores, scores)
