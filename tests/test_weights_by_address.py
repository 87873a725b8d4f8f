"""A pass names its weights, ids and scores to the native sequences by address.  Whatever layout a tensor has at that moment, the
address is that of its elements in order, and another number of elements is refused, also where a weight gradient is given its
place (CPU: the sequences are replaced by a recorder that reads the elements as the kernels would)."""

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


# Where a weight gradient goes: a GEMM writes every expert's part, so a parameter of another size is refused before anything is allocated
# or launched, also for MXFP8, whose source weights are not looked at after the forward.
SHAPE = (4, 6, 8)
CONFIG = types.SimpleNamespace(wgrad_dtype=None)  # of `_destination`


def _destination(param, explicit=None, **options):
    return _bf16._wgrad_destination(param, SHAPE, ExecutionOptions(**options), CONFIG, None, explicit)


@pytest.mark.parametrize("shape", [(2, 6, 8), (5, 6, 8), (4, 2, 3, 4)])
@pytest.mark.parametrize("how", ["fresh", "dtype", "tensor", "accumulate"])
def test_another_size_is_refused(shape, how):
    param = torch.zeros(shape, dtype=torch.bfloat16)
    explicit = {"dtype": torch.float32, "tensor": torch.zeros(shape)}.get(how)
    with pytest.raises(RuntimeError):
        _destination(param, explicit, inplace_wgrad_accum=how == "accumulate")
    assert param.grad is None


@pytest.mark.parametrize("shape", [(4, 6, 8), (4, 2, 3, 8), (24, 8)])
def test_the_same_size_in_any_shape(shape):
    param = torch.zeros(shape, dtype=torch.bfloat16)
    dst, accumulate, returned = _destination(param)
    assert dst.shape == param.shape and dst.is_contiguous() and (accumulate, returned) == (0, True)
    assert _destination(param, torch.float32)[0].dtype is torch.float32
    own = torch.zeros(shape)
    assert _destination(param, own)[0] is own
    assert _destination(param, inplace_wgrad_accum=True)[0] is param.grad
