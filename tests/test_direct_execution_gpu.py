"""BF16 training calls run the registered operators' bodies directly where nothing acts on operators.  The same call under
a dispatch mode goes through the operators; outputs and gradients are equal bit for bit."""

import contextlib

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import dist_moe_b200 as dm

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
T, D, F, E, K = 33, 192, 256, 6, 2


class _Watch(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if func.namespace == "dist_moe":
            self.seen.append(func._opname)
        return func(*args, **(kwargs or {}))


def _run(mode, *, ids=torch.int64, scores=torch.float32, accumulate=False, grad=torch.bfloat16, slots=None, norm=False,
         clamped=False, frozen=(), wrap=None, two_layers=False):
    g = torch.Generator().manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    x = rnd(T, D).bfloat16().to(DEV).requires_grad_("x" not in frozen)
    w13 = (rnd(E, 2, F, D) * D ** -0.5).bfloat16().to(DEV).requires_grad_("w13" not in frozen)
    w2 = (rnd(E, D, F) * F ** -0.5).bfloat16().to(DEV).requires_grad_("w2" not in frozen)
    top = torch.topk(rnd(T, E), K)
    s = torch.softmax(top.values, -1).to(scores).to(DEV).requires_grad_("scores" not in frozen)
    i = top.indices.to(ids).to(DEV)
    extra = dict(activation="swiglu_clamped", swiglu_limit=7.0) if clamped else {}
    if slots:
        extra["activation_slot_capacity_factor"] = slots
    cfg = dm.Config(max_num_local_input_tokens=T, hidden_dim=D, intermediate_dim=F, top_k=K, num_experts=E,
                    max_moe_layers_per_activation_slot=2 if two_layers else 1, wgrad_dtype=grad, **extra)
    post = dm.RMSNormPostprocess(eps=1e-6, norm_output_dtype=torch.float32, output_dtype=torch.bfloat16) if norm else None
    options = dm.ExecutionOptions(inplace_wgrad_accum=accumulate, experts_output_postprocess=post)
    if accumulate:
        for w in (w13, w2):
            if grad != w.dtype:
                w.grad_dtype = grad
            w.grad = torch.full(w.shape, 0.5, device=DEV, dtype=grad)
    context = dm.create_context(group=None, config=cfg, device=DEV)
    try:
        call = lambda a, b: dm.routed_experts(a, i, b, w13, w2, context, options=options)  # noqa: E731
        with mode:
            out = wrap(call, x, s) if wrap else call(x, s)
            out.backward(rnd(T, D).bfloat16().to(DEV))
        context.check_status()
        return [t.detach().clone() for t in (out, x.grad, s.grad, w13.grad, w2.grad) if t is not None]
    finally:
        context.close()


FORMS = [dict(), dict(ids=torch.int32, scores=torch.bfloat16), dict(slots=1.0), dict(accumulate=True),
         dict(accumulate=True, grad=torch.float32, slots=1.0), dict(grad=torch.float32), dict(norm=True),
         dict(norm=True, slots=1.0, clamped=True), dict(frozen=("w13",)), dict(frozen=("x", "scores")),
         dict(frozen=("scores",), clamped=True), dict(frozen=("w13", "w2"))]


@pytest.mark.parametrize("form", FORMS, ids=[str(i) for i in range(len(FORMS))])
def test_direct_equals_operators(form):
    watch = _Watch()
    through = _run(watch, **form)
    assert len(watch.seen) == 2 and watch.seen[0] == "bf16_forward", watch.seen
    direct = _run(contextlib.nullcontext(), **form)
    assert len(direct) == len(through)
    for a, b in zip(direct, through):
        assert a.dtype == b.dtype and torch.equal(a, b)


def test_saved_tensors_may_move():
    plain = _run(contextlib.nullcontext())
    for a, b in zip(_run(torch.autograd.graph.save_on_cpu()), plain):
        assert torch.equal(a, b)


def test_a_mode_that_ends_before_the_backward():
    """The forward through the operators, the backward outside the mode, and the other way round."""
    plain = _run(contextlib.nullcontext())

    def forward_watched(call, x, s):
        with _Watch() as watch:
            out = call(x, s)
        assert watch.seen == ["bf16_forward"]
        return out

    for a, b in zip(_run(contextlib.nullcontext(), wrap=forward_watched), plain):
        assert torch.equal(a, b)

    class Late(contextlib.nullcontext):
        pass

    watch = _Watch()
    late = Late()

    def enter_after(call, x, s):
        out = call(x, s)
        late.stack = contextlib.ExitStack()
        late.stack.enter_context(watch)
        return out

    try:
        for a, b in zip(_run(late, wrap=enter_after), plain):
            assert torch.equal(a, b)
    finally:
        late.stack.close()
    assert watch.seen == ["bf16_backward"]


def test_a_differentiated_backward_is_refused():
    cfg = dm.Config(max_num_local_input_tokens=T, hidden_dim=D, intermediate_dim=F, top_k=K, num_experts=E,
                    max_moe_layers_per_activation_slot=1)
    context = dm.create_context(group=None, config=cfg, device=DEV)
    try:
        x = torch.randn(T, D, device=DEV).bfloat16().requires_grad_()
        w13 = torch.randn(E, 2, F, D, device=DEV).bfloat16().requires_grad_()
        w2 = torch.randn(E, D, F, device=DEV).bfloat16().requires_grad_()
        ids = torch.arange(T * K, device=DEV).reshape(T, K) % E
        out = dm.routed_experts(x, ids, torch.full((T, K), 0.5, device=DEV), w13, w2, context)
        (gx,) = torch.autograd.grad(out.float().sum(), x, create_graph=True)
        with pytest.raises(RuntimeError):
            gx.float().sum().backward()
    finally:
        context.close()


@pytest.mark.parametrize("form", [dict(), dict(slots=1.0), dict(norm=True)], ids=["plain", "saved", "norm"])
@pytest.mark.parametrize("watched", ["forward", "backward", "both"])
def test_checkpointing_under_modes(form, watched):
    """Non-reentrant checkpointing compares the tensors that a forward and its repetition save, also where a mode covers only
    one of them."""
    from torch.utils.checkpoint import checkpoint

    plain = _run(contextlib.nullcontext(), **form)
    stack = contextlib.ExitStack()

    def call_checkpointed(call, x, s):
        with _Watch() if watched in ("forward", "both") else contextlib.nullcontext():
            out = checkpoint(call, x, s, use_reentrant=False)
        if watched in ("backward", "both"):
            stack.enter_context(_Watch())
        return out

    with stack:
        got = _run(contextlib.nullcontext(), wrap=call_checkpointed, two_layers=True, **form)
    for a, b in zip(got, plain):
        assert torch.equal(a, b)
