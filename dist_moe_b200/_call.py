"""What the BF16 and the MXFP8 training passes share on the host: the device results of a call, the argument structure of the
native launch sequences, and running their steps.

A pass is one or two native calls (``dm_bf16_forward`` and the like, csrc/sequence.cu); only observed passes (a profiler's
ranges, GEMMs timed in place) and passes with Python callbacks between launches take more.  A foreign-function call per
launch, a tensor per result and the dispatcher around the registered operators made small layers wait for the host: forward and
backward of 16 tokens (D = F = 256, 8 experts) 656 -> 301 us, of 1531 tokens (D = 1088, F = 704, 24 experts, recomputed) 674 ->
330 us, MXFP8 of 777 tokens with tensor weights 580 -> 397 us.
What was left in Python (views and detached copies of tensors whose address alone was used, the layout of a call's results laid
out twice per pass, device guards for the device that is current, imports inside functions) took 50 of 147 us of the first: 294 ->
249 us; MXFP8 of 777 tokens 388 -> 351.
"""

from __future__ import annotations

import ctypes
import os
import sys

import torch
from torch.profiler import record_function

from . import _native as nat

# Steps of the forward and backward sequences (include/dist_moe_b200.h), in launch order.
FWD = {name: 1 << i for i, name in enumerate(
    ("publish", "route", "save_x", "w13", "swiglu", "w2", "combine", "reduce"))}
BWD = {name: 1 << i for i, name in enumerate(
    ("plan", "republish", "w13_again", "swiglu_again", "w2_again", "load_h3", "grad_h3", "combine", "w2_dgrad", "w2_wgrad",
     "swiglu", "w13_dgrad", "w13_wgrad", "close", "reduce"))}
FWD_ALL = 255
_TIMED = {
    "dm_bf16_forward": {"w13": "gemm_fprop_dispatch(w13)", "w2": "gemm_fprop(w2)"},
    "dm_bf16_backward": {
        "w13_again": "gemm_fprop_dispatch(w13 recompute)", "w2_again": "gemm_fprop(w2 recompute)",
        "w2_dgrad": "gemm_dgrad_dispatch(w2)", "w2_wgrad": "gemm_wgrad(w2)", "w13_dgrad": "gemm_dgrad(w13)",
        "w13_wgrad": "gemm_wgrad(w13)"},
    "dm_mxfp8_forward": {name: f"forward.{name}" for name in FWD},
    "dm_mxfp8_backward": {name: f"backward.{name}" for name in BWD},
}
_REPORT = ctypes.c_int32 * 2


def _recorder_query():
    """``at::hasCallbacks()`` of ATen/record_function.h, which Python does not bind: whether anything records operators and
    ranges on this thread.  That is the profiler, but also an ``ExecutionTraceObserver`` or NVTX emission, which
    ``torch.autograd._profiler_enabled`` does not know of.  0.1 us a call; where the symbol is missing, always."""
    try:
        query = ctypes.PyDLL(os.path.join(os.path.dirname(torch.__file__), "lib", "libtorch_cpu.so"))._ZN2at12hasCallbacksEv
    except (OSError, AttributeError):
        return lambda: True
    query.restype, query.argtypes = ctypes.c_bool, []
    return query


recorded = _recorder_query()


def _profile() -> list | None:
    """``_bf16.PROFILE`` of this moment (that module imports this one)."""
    bf16 = sys.modules.get(_BF16)
    return None if bf16 is None else bf16.PROFILE


_BF16 = __package__ + "._bf16"


def observed() -> bool:
    """Someone wants to see the parts of a pass."""
    return _profile() is not None or recorded()


class _NoSpan:
    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False


_NOTHING = _NoSpan()


def span(name: str):
    """A profiler range with the reference's name (dist_moe/api.py:1979-2443), free where nothing records."""
    return record_function(name) if recorded() else _NOTHING


def on_device(device: torch.device):
    """``torch.cuda.device``, free where the device is the current one already."""
    return _NOTHING if torch._C._cuda_getDevice() == device.index else torch.cuda.device(device)


def launch(fn, names: dict, state, k, steps: int) -> None:
    """Run the given steps of a sequence: one call, or one per step where they are timed in place."""
    context, st = state.native_layer(), nat.stream_ptr()

    def run(bits: int) -> None:
        report = _REPORT()
        rc = fn(context, ctypes.byref(k), bits, report, st)
        nat.LAUNCHES[0] += report[0]
        if rc != 0:
            failed = next((n for n, bit in names.items() if bit == report[1]), "arguments")
            nat.check(rc, f"{fn.__name__}({failed})")

    profile = _profile()
    if profile is None:
        run(steps)
        return
    timed = _TIMED[fn.__name__]
    for name, bit in names.items():
        if not steps & bit:
            continue
        if name not in timed:
            run(bit)
            continue
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        run(bit)
        end.record()
        profile.append((timed[name], start, end))


def in_one_piece(t: torch.Tensor, numel: int, name: str) -> torch.Tensor:
    """``t``, or a contiguous copy of it, for a pass that uses the address alone.  Checks at the entry point do not cover this: there
    a weight's dimensions are merged first, which copies a (E, 2, F, D) view whose leading dimensions do not merge, and what a
    backward unpacks is the leaf as it is at that moment (its ``.data`` may have been replaced) or what a saved-tensor hook made of
    it.  The caller keeps the result alive until the pass is launched."""
    if t.numel() != numel:
        raise RuntimeError(f"{name} has {numel} elements in this call, not {t.numel()} (shape {tuple(t.shape)})")
    return t if t.is_contiguous() else t.detach().contiguous()


def routes_in_one_piece(ids: torch.Tensor, scores: torch.Tensor, routes: int) -> tuple[torch.Tensor, torch.Tensor]:
    if ids.numel() == routes == scores.numel() and ids.is_contiguous() and scores.is_contiguous():
        return ids, scores
    return in_one_piece(ids, routes, "topk_expert_ids_TK"), in_one_piece(scores, routes, "topk_scores_TK")


class Layout:
    """Where the device results of a call lie in their buffer.  ``fields``: name -> (dtype, elements)."""

    def __init__(self, fields: dict):
        self.fields, self.at, off = fields, {}, 0
        for name, (dtype, n) in fields.items():
            self.at[name] = off
            off += (n * dtype.itemsize + 15) & ~15
        self.words = off // 8


def layout_of(state, key: tuple, fields) -> Layout:
    """The layout of this kind of call, built by ``fields()`` unless the context's last call was of the same kind."""
    last = getattr(state, "_call_layout", None)
    if last is None or last[0] != key:
        last = state._call_layout = (key, Layout(fields()))  # one assignment: threads may call in turn
    return last[1]


class CallState:
    """Device results of routing and planning of one call: one buffer (``buf``) that the names of the layout are views of, or
    tensors of their own where a registered operator hands them out."""

    def __init__(self, layout: Layout):
        self.fields, self.at, self.words, self.buf = layout.fields, layout.at, layout.words, None
        self.rstd = self.callback_state = None

    def allocate(self, device, separate: bool = False) -> "CallState":
        if separate:
            for name, (dtype, n) in self.fields.items():
                setattr(self, name, torch.empty(n, dtype=dtype, device=device) if n else None)
        else:
            self.buf = torch.empty(self.words, dtype=torch.int64, device=device)
        return self

    def adopt(self, buf: torch.Tensor) -> "CallState":
        """The results that an earlier call has left in ``buf``."""
        self.buf = buf
        return self

    def ptr(self, name: str) -> int | None:
        if self.buf is None:
            return nat.ptr(getattr(self, name))
        return self.buf.data_ptr() + self.at[name] if self.fields[name][1] else None

    def __getattr__(self, name: str):  # views of the buffer, made when asked for
        if name == "recv_rows":
            return self.offsets[self.offsets.numel() - 1:]
        fields = self.__dict__.get("fields", {})
        if name not in fields or self.__dict__.get("buf") is None:
            raise AttributeError(name)
        dtype, n = fields[name]
        at = self.at[name]
        view = self.buf.view(torch.uint8)[at:at + n * dtype.itemsize].view(dtype) if n else None
        setattr(self, name, view)
        return view


def arguments(state, c: CallState, x, ids, scores, options) -> "nat.LayerCall":
    """What the passes of a call have in common."""
    k = nat.LayerCall()
    if x is not None:
        k.x = x.data_ptr()
    k.ids, k.ids_are_int64 = ids.data_ptr(), ids.dtype is torch.int64
    k.scores, k.scores_are_bf16 = scores.data_ptr(), scores.dtype is torch.bfloat16
    if c.buf is None:
        ptr = c.ptr
        k.counts, k.per_rank, k.expert_offsets = ptr("counts"), ptr("per_rank"), ptr("offsets")
        k.fwd_ptrs, k.bwd_ptrs, k.sct_ptrs = ptr("fwd"), ptr("bwd"), ptr("sct")
        k.need, k.cond, k.fwd_state = ptr("need"), ptr("cond"), ptr("fwd_state")
    else:
        base, at = c.buf.data_ptr(), c.at
        k.counts, k.per_rank, k.expert_offsets = base + at["counts"], base + at["per_rank"], base + at["offsets"]
        k.fwd_ptrs, k.sct_ptrs = base + at["fwd"], base + at["sct"]
        k.bwd_ptrs = base + at["bwd"] if c.fields["bwd"][1] else None
        k.need, k.cond, k.fwd_state = base + at["need"], base + at["cond"], base + at["fwd_state"]
    k.T, k.ptrs_size, k.max_rows = c.T, c.size, c.max_rows
    k.num_layers, k.validate_ids = state.num_layers_in_slot, options.validate_expert_ids
    return k
