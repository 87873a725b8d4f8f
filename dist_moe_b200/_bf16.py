"""BF16 routed-expert forward and backward: kernel sequencing and autograd glue.

Launch order follows the reference's BF16 orchestration
(dist_moe/api.py:1844-2188 forward, 2205-2609 backward):

forward   publish -> barrier -> route -> plan -> [save x] -> gather -> W13 (+SwiGLU) ->
          W2 + scatter -> barrier -> weighted top-k reduce (+ save h3)
backward  plan -> [recompute: republish, barrier, gather, W13, SwiGLU, W2 + scatter] ->
          grad_h3 / grad_scores -> barrier -> gather grad_h3 + W2 dgrad -> W2 wgrad ->
          SwiGLU bwd -> W13 dgrad + scatter -> W13 wgrad -> barrier -> reduce

Every data-dependent decision (row counts, arena offsets, save-versus-recompute) stays
on the device: the host never reads a device value, so the sequence can be captured in a
CUDA graph.  Bracketed steps are device-predicated on the planner's decision.
"""

from __future__ import annotations

from typing import Any

import torch

from . import _native as nat
from ._call import (BWD, FWD, FWD_ALL, CallState, Layout, arguments, in_one_piece, launch, layout_of, observed, on_device,
                    recorded, routes_in_one_piece, span)
from ._execution import ExecutionOptions, RMSNormPostprocess


# When set to a list, every grouped-GEMM launch of a BF16 pass and every step of an MXFP8 training pass is bracketed by
# CUDA events on the launching stream and (name, start, end) is appended; benchmarks use it to time the kernels in place.
PROFILE: list | None = None

# Fused dispatch pulls the routed rows inside the W13 / W2-dgrad GEMM launches (gather warps overlap the peer
# transfer with the tensor cores).  With False the rows are gathered by a separate kernel first.
FUSED_DISPATCH = True
# The plain backward reads saved expert outputs where they were saved (chosen on the device) instead of copying
# them back into the communication buffer first.  False restores the copy.
READ_SAVED_H3_IN_PLACE = True


class _Call(CallState):
    """Device results of routing and planning of one BF16 call."""

    def __init__(self, state=None, T: int = 0, with_bwd: bool = True):
        if state is None:
            super().__init__(Layout({}))
            return
        el, size = state.e_local, state.ep * state.e_local * T

        def fields():
            i64, i32 = torch.int64, torch.int32
            return {"fwd_state": (i64, 6), "need": (torch.uint8, 1), "cond": (i32, 1), "counts": (i32, el),
                    "per_rank": (i32, state.ep), "offsets": (i32, el + 1), "fwd": (i64, size), "sct": (i64, size),
                    "bwd": (i64, size if with_bwd else 0), "bwd_offsets": (i64, 6 if with_bwd else 0)}

        super().__init__(layout_of(state, ("bf16", T, with_bwd), fields))
        self.T, self.size, self.max_rows = T, size, min(size, state.capacity_rows)

    def saved(self) -> list[torch.Tensor]:
        """The state list of the registered operators, as views of the buffer."""
        at, words, halves = self.at, self.buf, self.buf.view(torch.int32)

        def piece(name: str, of: torch.Tensor, size: int, first: int = 0) -> torch.Tensor:
            start = at[name] // size
            return of[start + first:start + self.fields[name][1]]

        rstd = self.rstd if self.rstd is not None else torch.empty(0, dtype=torch.float32, device=words.device)
        return [piece("counts", halves, 4), piece("bwd", words, 8), piece("fwd", words, 8), piece("sct", words, 8),
                piece("per_rank", halves, 4), piece("offsets", halves, 4, self.fields["counts"][1]),
                words[at["need"] // 8:].view(torch.uint8)[:1], piece("fwd_state", words, 8), rstd]

    @staticmethod
    def from_saved(state, tensors: list[torch.Tensor], T: int):
        """The call whose ``saved`` tensors these are, or None: they may be an operator's, or hooks have put them elsewhere."""
        c = _Call(state, T)
        total, storage = c.words, tensors[7].untyped_storage()
        if storage.nbytes() != 8 * total:
            return None
        at, base = c.at, storage.data_ptr()
        places = (at["counts"], at["bwd"], at["fwd"], at["sct"], at["per_rank"], at["offsets"] + 4 * state.e_local, at["need"],
                  at["fwd_state"])
        if any(t.data_ptr() != base + place for t, place in zip(tensors, places)):
            return None
        c.adopt(tensors[7].as_strided((total,), (1,), 0))
        c.rstd = tensors[8] if tensors[8].numel() else None
        return c


def _arguments(state, c: _Call, x, ids, scores, w13, w2, options: ExecutionOptions, scratch_only: bool):
    k = arguments(state, c, x, ids, scores, options)
    k.w13, k.w2 = w13.data_ptr(), w2.data_ptr()
    k.scratch_only, k.separate_gather = scratch_only, not FUSED_DISPATCH
    return k


def _weights_in_one_piece(state, w13, w2):
    cfg = state.config
    n = state.e_local * cfg.intermediate_dim * cfg.hidden_dim
    if w2.numel() == n and w13.numel() == 2 * n and w2.is_contiguous() and w13.is_contiguous():
        return w13, w2
    return in_one_piece(w13, 2 * n, "w13"), in_one_piece(w2, n, "w2")


def _forward(state, k, steps: int) -> None:
    launch(nat.lib.dm_bf16_forward, FWD, state, k, steps)


def _backward(state, k, steps: int) -> None:
    launch(nat.lib.dm_bf16_backward, BWD, state, k, steps)


def forward_impl(state, x, ids, scores, w13, w2, options: ExecutionOptions, save_for_backward: bool, hooks=None,
                 separate: bool = False):
    """``separate``: the call's device results as tensors of their own (registered operators return them)."""
    cfg = state.config
    T, F = x.shape[0], cfg.intermediate_dim
    w13, w2 = _weights_in_one_piece(state, w13, w2)
    scratch_only = (not save_for_backward) or cfg.inference or state.num_slots == 0
    c = _Call(state, T, not scratch_only).allocate(x.device, separate)
    out = torch.empty(x.shape, dtype=torch.bfloat16, device=x.device)
    k = _arguments(state, c, x, ids, scores, w13, w2, options, scratch_only)
    k.out = out.data_ptr()
    clip = options.swiglu_clip_stats_out_3
    if clip is not None:
        clip.zero_()
        k.clip_stats, k.clip_limit = clip.data_ptr(), float(options.swiglu_clip_limit)
    k.fuse_swiglu = clip is None and F % 128 == 0
    post = options.experts_output_postprocess
    state.last_call = c
    if not observed():
        _forward(state, k, FWD_ALL if post is None else FWD_ALL - FWD["reduce"])
    else:
        with span("dist_moe_routing"):
            with span("dist_moe_preprocess"):  # publish ids and rows, then the barrier every peer waits on
                _forward(state, k, FWD["publish"])
            _forward(state, k, FWD["route"])
        _forward(state, k, FWD["save_x"])
        with span("dist_moe_forward"):
            _forward(state, k, FWD["w13"] | FWD["swiglu"] | FWD["w2"])
        _forward(state, k, FWD["combine"] | (FWD["reduce"] if post is None else 0))
    if isinstance(post, RMSNormPostprocess):
        from ._postprocess import rmsnorm_combine_forward

        if hooks is not None:
            hooks.observe_expert_output(state, post, ids, T)
        c.rstd = rmsnorm_combine_forward(state, c, post, scores, ids, out, save=not scratch_only,
                                         observers_allowed=hooks is not None)
    elif post is not None:
        if hooks is None:
            raise RuntimeError("a callable expert-output post-process runs on the eager path only")
        hooks.postprocess_forward(state, c, post, scores, ids, out, save=not scratch_only)
    return out, c


def _wgrad_destination(param: torch.Tensor, shape, options: ExecutionOptions, cfg, owner: torch.Tensor | None,
                       explicit=None, hooks=None, name: str = ""):
    """Return (tensor, accumulate, returned_to_autograd).

    ``explicit`` is used by the registered operators: a tensor to accumulate into, or a dtype for a fresh result.
    ``hooks`` (eager path) may name the destination through ``wgrad_destination_fn``.
    """
    if hooks is not None:
        named = hooks.wgrad_destination(name, shape, cfg.wgrad_dtype or param.dtype, param.device)
        if named is not None:
            return named[0], int(named[1]), False
    if param.numel() != shape[0] * shape[1] * shape[2]:  # the weight may be another one by now than in the forward; a GEMM writes all of ``shape``
        raise RuntimeError(f"the gradient of a weight of shape {tuple(param.shape)} cannot hold one of shape {tuple(shape)}")
    if isinstance(explicit, torch.Tensor):
        if not explicit.is_contiguous() or explicit.dtype not in (torch.bfloat16, torch.float32) \
                or explicit.numel() != param.numel():
            raise ValueError("WGRAD accumulators must be contiguous BF16 or FP32 tensors of the weight's size")
        return explicit, 1, False
    if isinstance(explicit, torch.dtype):
        if explicit not in (torch.bfloat16, torch.float32):
            raise ValueError("wgrad_output_dtype must be torch.bfloat16 or torch.float32")
        return torch.empty(param.shape, dtype=explicit, device=param.device), 0, True
    if options.inplace_wgrad_accum:
        target = owner if owner is not None else param
        if target.grad is None:
            dtype = cfg.wgrad_dtype or getattr(target, "grad_dtype", None) or target.dtype
            if dtype != target.dtype and hasattr(target, "grad_dtype"):
                target.grad_dtype = dtype
            target.grad = torch.zeros_like(target, dtype=dtype)
        grad = target.grad
        if not grad.is_contiguous() or grad.dtype not in (torch.bfloat16, torch.float32):
            raise ValueError("in-place WGRAD accumulation needs a contiguous BF16 or FP32 parameter.grad")
        if grad.numel() != param.numel():
            raise ValueError("WGRAD owner gradient does not match the compute weight size")
        return grad, 1, False
    dtype = cfg.wgrad_dtype or param.dtype
    return torch.empty(param.shape, dtype=dtype, device=param.device), 0, True


def backward_impl(state, c: _Call, x_shape, ids, scores, w13, w2, w13_param, w2_param, grad_out,
                  options: ExecutionOptions, needs, wgrad_explicit=(None, None), hooks=None):
    cfg = state.config
    T, D, K, F, el = c.T, cfg.hidden_dim, cfg.top_k, cfg.intermediate_dim, state.e_local
    dev = grad_out.device
    need_x, need_scores, need_w13, need_w2 = needs
    w13, w2 = _weights_in_one_piece(state, w13, w2)
    ids, scores = routes_in_one_piece(ids, scores, T * K)
    # the plan's offsets: [xg, h1, h2, grad_h2, grad_h3_gathered, grad_h1]
    bo = torch.empty(6, dtype=torch.int64, device=dev) if c.buf is None else None
    grad_scores = torch.empty(T, K, dtype=torch.float32, device=dev) if need_scores else None
    post = options.experts_output_postprocess
    is_norm = isinstance(post, RMSNormPostprocess)
    is_callback = post is not None and not is_norm  # the callable kept its own input and output (eager path)
    k = _arguments(state, c, None, ids, scores, w13, w2, options, False)
    k.bwd_offsets, k.grad_out, k.grad_scores = c.ptr("bwd_offsets") if bo is None else bo.data_ptr(), grad_out.data_ptr(), nat.ptr(grad_scores)
    # Saved expert outputs: the fused RMSNorm backward works on them in place in the communication buffer, so they are
    # copied back there; the plain backward reads them where they were saved (selected on the device).
    load_h3 = is_norm or (need_scores and not is_callback and not READ_SAVED_H3_IN_PLACE)
    k.h3_in_combine = load_h3
    # recompute block: every launch is a no-op unless the forward chose to recompute this layer; h2 is always rebuilt
    recompute = BWD["plan"] | BWD["republish"] | BWD["w13_again"] | BWD["swiglu_again"]
    if (need_scores or is_norm) and not is_callback:
        recompute |= BWD["w2_again"] | (BWD["load_h3"] if load_h3 else 0)
    first = 0 if observed() or post is not None else recompute | BWD["grad_h3"] | BWD["combine"] | BWD["w2_dgrad"]
    if first == 0:
        with span("dist_moe_recompute"):
            _backward(state, k, recompute)
    with span("dist_moe_backward"):
        # ---- grad wrt expert outputs and scores ------------------------------------
        if is_norm:
            from ._postprocess import rmsnorm_combine_backward

            kept = None
            if hooks is not None:
                # the replay of a recomputed layer shows its expert outputs to the forward observer again; whether the
                # layer was recomputed is a device-side decision, read here because observers run on the host anyway
                if post.observe_expert_output_fn is not None and bool(c.need.item()):
                    hooks.observe_expert_output(state, post, ids, T)
                kept = hooks.preserved_expert_output(state, post, ids, T)
            rmsnorm_combine_backward(state, c, post, grad_out, scores, ids, grad_scores, h3=kept)
            if kept is not None:
                hooks.observe_expert_output_grad(state, post, kept, T)
        elif is_callback:
            hooks.postprocess_backward(state, c, grad_out, scores, ids, grad_scores)
        rest = BWD["combine"] | BWD["w2_dgrad"] | (BWD["grad_h3"] if post is None else 0)
        _backward(state, k, first if first else rest)
        # ---- W2 weight gradient; SwiGLU backward, W13 input gradient (scattered to the owners) and weight gradient ----
        grad_w13 = grad_w2 = grad_x = None
        owners = options.wgrad_parameter_owners or (None, None)
        steps = 0
        if need_w2:
            dst, k.dw2_accumulate, ret = _wgrad_destination(w2_param, (el, D, F), options, cfg, owners[1],
                                                            wgrad_explicit[1], hooks, "w2")
            k.dw2, k.dw2_is_fp32 = dst.data_ptr(), dst.dtype is torch.float32
            grad_w2 = dst if ret else None
            steps = BWD["w2_wgrad"]
            if hooks is not None:
                _backward(state, k, steps)
                grad_w2, steps = hooks.wgrad_postprocess("w2", grad_w2), 0
        steps |= BWD["swiglu"]
        if need_x:
            steps |= BWD["w13_dgrad"]
        if need_w13:
            if hooks is not None:  # named destinations are asked for when the gradient is next
                _backward(state, k, steps)
                steps = 0
            dst, k.dw13_accumulate, ret = _wgrad_destination(w13_param, (el, 2 * F, D), options, cfg, owners[0],
                                                             wgrad_explicit[0], hooks, "w13")
            k.dw13, k.dw13_is_fp32 = dst.data_ptr(), dst.dtype is torch.float32
            grad_w13 = dst if ret else None
            steps |= BWD["w13_wgrad"]
            if hooks is not None:
                _backward(state, k, steps)
                grad_w13, steps = hooks.wgrad_postprocess("w13", grad_w13), 0
        steps |= BWD["close"]
        if need_x:
            grad_x = torch.empty(x_shape, dtype=torch.bfloat16, device=dev)
            k.grad_x = grad_x.data_ptr()
            steps |= BWD["reduce"]
        _backward(state, k, steps)
        if grad_scores is not None and scores.dtype != torch.float32:
            grad_scores = grad_scores.to(scores.dtype)
    return grad_x, grad_scores, grad_w13, grad_w2


class _Bf16Function(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, ids, scores, w13_param, w2_param, state, options):
        cfg = state.config
        w13 = w13_param.detach().reshape(state.e_local, 2 * cfg.intermediate_dim, cfg.hidden_dim)
        w2 = w2_param.detach().reshape(state.e_local, cfg.hidden_dim, cfg.intermediate_dim)
        out, call = forward_impl(state, x.detach(), ids, scores.detach(), w13, w2, options, True)
        ctx.state, ctx.call, ctx.options = state, call, options
        ctx.x_shape = x.shape
        ctx.save_for_backward(ids, scores, w13_param, w2_param)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        ids, scores, w13_param, w2_param = ctx.saved_tensors
        state, cfg = ctx.state, ctx.state.config
        w13 = w13_param.detach().reshape(state.e_local, 2 * cfg.intermediate_dim, cfg.hidden_dim)
        w2 = w2_param.detach().reshape(state.e_local, cfg.hidden_dim, cfg.intermediate_dim)
        needs = (ctx.needs_input_grad[0], ctx.needs_input_grad[2], ctx.needs_input_grad[3], ctx.needs_input_grad[4])
        with torch.cuda.device(state.device):
            gx, gs, gw13, gw2 = backward_impl(state, ctx.call, ctx.x_shape, ids, scores.detach(), w13, w2, w13_param,
                                              w2_param, grad_out.contiguous(), ctx.options, needs)
        return gx, None, gs, gw13, gw2, None, None


def _rmsnorm_args(post):
    """The RMSNorm arguments of the registered operators (weight, enabled, eps, norm dtype, output dtype, bitwise,
    gain centre, Kahan, recompute rstd); disabled values when there is no RMSNorm post-process."""
    if isinstance(post, RMSNormPostprocess):
        return (post.weight, True, float(post.eps), post.norm_output_dtype, post.output_dtype, bool(post.require_bitwise),
                float(post.gain_center), bool(post.use_kahan), bool(post.recompute_rstd))
    return (None, False, 1e-6, torch.float32, torch.bfloat16, False, 0.0, False, False)


def _plain_execution(*tensors) -> bool:
    """Nothing acts on this call's operators: no tracing or fake tensors, no dispatch or function mode, no functorch
    level, no recorder (profiler, execution trace).  The registered operators' bodies can then run without the dispatcher,
    which costs a small layer more than its launches."""
    if torch.compiler.is_compiling():  # first: a tracer of Python code must not meet the calls below
        return False
    for t in tensors:
        kind = type(t)
        if kind is not torch.Tensor and kind is not torch.nn.Parameter:
            return False
    c = torch._C
    return (not recorded() and c._len_torch_dispatch_stack() == 0 and c._len_torch_function_stack() == 0
            and torch._ops._len_torch_dispatch_stack_pre_dispatch() == 0
            and c._functorch.peek_interpreter_stack() is None and c._get_tracing_state() is None)


class _RegisteredBf16Function(torch.autograd.Function):
    """Training call through the registered operators ``dist_moe::bf16_forward`` (``..._with_clip_stats``) and
    ``dist_moe::bf16_backward`` / ``bf16_backward_accumulate_`` (dist_moe/api.py:4027-4042 applies its
    ``_RegisteredBf16Autograd`` the same way), so that FakeTensor propagation, ``make_fx`` and ``torch.compile`` of
    the caller's code see operator nodes with the reference's names and schemas.  Where nothing acts on operators
    (``_plain_execution``) their bodies run directly, with the call's device results in one buffer."""

    @staticmethod
    def forward(ctx, x, ids, scores, w13_param, w2_param, context, options):
        state = context._state
        clip = options.swiglu_clip_stats_out_3
        ctx.context, ctx.options = context, options
        if clip is None and _plain_execution(x, ids, scores, w13_param, w2_param):
            # gradients are off here
            out, call = forward_impl(state, x, ids, scores, w13_param, w2_param, options, True)
            # What a call saves must not depend on the way it goes where saved-tensor hooks look at it: activation
            # checkpointing compares a forward with its repetition, which may run under other modes.
            hooked = torch._C._autograd._top_saved_tensors_default_hooks(False) is not None
            ctx.save_for_backward(ids, scores, w13_param, w2_param, *(call.saved() if hooked else (call.buf, call.rstd)))
            return out
        rms = _rmsnorm_args(options.experts_output_postprocess)
        head = (x.detach().contiguous(), ids, scores.detach(), w13_param.detach(), w2_param.detach(), *rms,
                state.slot_selector, state.num_layers_in_slot, bool(options.validate_expert_ids))
        if clip is None:
            out, st = torch.ops.dist_moe.bf16_forward(*head, context._context_id)
        else:
            out, st, counters = torch.ops.dist_moe.bf16_forward_with_clip_stats(*head, float(options.swiglu_clip_limit),
                                                                                  context._context_id)
            clip.copy_(counters)  # graph-visible copy into the caller's tensor
        ctx.save_for_backward(ids, scores, w13_param, w2_param, *st)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        ids, scores, w13_param, w2_param, *st = ctx.saved_tensors
        context, options = ctx.context, ctx.options
        cfg, state = context.config, context._state
        need = ctx.needs_input_grad
        needs = (need[0], need[2], need[3], need[4])
        e_local, D, F = state.e_local, cfg.hidden_dim, cfg.intermediate_dim
        destinations = (cfg.wgrad_dtype or w13_param.dtype,) * 2
        if options.inplace_wgrad_accum:
            owners = options.wgrad_parameter_owners or (None, None)
            destinations = (_wgrad_destination(w13_param, (e_local, 2 * F, D), options, cfg, owners[0])[0],
                            _wgrad_destination(w2_param, (e_local, D, F), options, cfg, owners[1])[0])
        whole = None
        if len(st) == 2:
            whole = _Call(state, ids.shape[0]).adopt(st[0])
            whole.rstd = st[1]
        # a backward that is itself differentiated goes through the operators, which refuse it
        if not torch.is_grad_enabled() and _plain_execution(grad_out, ids, scores, w13_param, w2_param, st[0]):
            if context._closed:
                raise RuntimeError(f"distributed MoE context {context._context_id} is not live")
            call = whole
            if call is None:
                from . import _ops

                call = _ops._unpack_bf16_state(state, st, ids.shape[0])
            with on_device(state.device):
                gx, gs, g13, g2 = backward_impl(state, call, grad_out.shape, ids, scores, w13_param, w2_param, w13_param,
                                                w2_param, grad_out.contiguous(), options, needs, destinations)
            if options.inplace_wgrad_accum:
                torch.autograd.graph.increment_version(destinations)  # as the operator's mutated arguments
            return gx, None, gs, g13, g2, None, None
        from . import _ops

        if whole is not None:
            st = whole.saved()
        rms = _rmsnorm_args(options.experts_output_postprocess)
        tail = (rms[1], rms[2], rms[3], rms[4], rms[5], rms[7], rms[8])
        _ops.NEEDS_HINT.append(needs)
        try:
            if options.inplace_wgrad_accum:
                gx, gs = torch.ops.dist_moe.bf16_backward_accumulate_(
                    grad_out.contiguous(), w13_param.detach(), w2_param.detach(), *destinations, ids, scores.detach(), st,
                    *tail, destinations[0].dtype, context._context_id)
                g13 = g2 = None
            else:
                gx, gs, g13, g2 = torch.ops.dist_moe.bf16_backward(
                    grad_out.contiguous(), w13_param.detach(), w2_param.detach(), ids, scores.detach(), st, *tail,
                    destinations[0], context._context_id)
        finally:
            _ops.NEEDS_HINT.clear()
        if gs is not None and needs[1] and gs.dtype != scores.dtype:
            gs = gs.to(scores.dtype)
        return (gx if needs[0] else None, None, gs if needs[1] else None, g13 if needs[2] else None,
                g2 if needs[3] else None, None, None)


def _registered_ops_are_ours() -> bool:
    from . import _ops

    return "bf16_forward" in _ops.REGISTERED


def run_bf16(x, ids, scores, w13_weight, w2_weight, w13_EFD, w2_EDF, context: Any, options: ExecutionOptions, *,
             save_for_backward: bool) -> torch.Tensor:
    state = context._state
    if options.requires_eager:
        from ._eager import run_bf16_eager

        return run_bf16_eager(x, ids, scores, w13_weight, w2_weight, context, options, save_for_backward=save_for_backward)
    if save_for_backward:
        if _registered_ops_are_ours():
            return _RegisteredBf16Function.apply(x, ids, scores, w13_weight, w2_weight, context, options)
        return _Bf16Function.apply(x, ids, scores, w13_weight, w2_weight, state, options)
    out, _ = forward_impl(state, x.detach(), ids, scores.detach(), w13_EFD.detach(), w2_EDF.detach(), options, False)
    return out
