"""Calls that break the last-in-first-out order of an activation slot: forwards without a backward, backwards out of order
or repeated.  The free pointer of the slot leaves it, in the end the arena; the bounded plan keeps every byte that a launch
touches inside the arena, whatever the order (oracle on the CPU, planner kernels and layers on the GPU)."""

import random

import pytest
import torch

from oracle import planner as bf16
from oracle import planner_blockscaled as bs

SLOTS, LAYERS, K, D, F, T = 2, 2, 2, 256, 384, 64
ROWS = 256  # most rows of a call
BOUNDED = 1 << 16  # DM_PLAN_BOUNDED


def _sizes(kind, rows):
    al, s = bf16.align, bs.MXFP8
    if kind == "bf16":
        return dict(x=al(T * D * 2), xg=al(rows * D * 2), h1=al(rows * 4 * F), h2=al(rows * 2 * F), h3=al(T * K * D * 2))
    return dict(x=al(T * D * 2), xg=sum(bs.col_sizes(rows, D, s)), h1=al(rows * 4 * F), h2=sum(bs.col_sizes(rows, F, s)),
                h3=al(T * K * D * 2))


def _scenario(kind, seed):
    """(slot bytes, arena bytes, operations): ("f", slot, rows) or ("b", index of the forward)."""
    rng = random.Random(seed)
    z = _sizes(kind, ROWS)
    full = z["xg"] + z["h1"] + z["h3"] + (z["h2"] if kind == "mxfp8" else 0)
    slot = bf16.align(int(LAYERS * z["x"] + rng.uniform(0, 1.2) * LAYERS * full))
    scratch = 6 * ROWS * (D + 2 * F)  # 1.6 MB: enough for any one call
    ops, forwards = [], 0
    for _ in range(150):
        if forwards and rng.random() < 0.25:
            ops.append(("b", rng.randrange(forwards)))  # any forward, also one that has had its backward
        else:
            ops.append(("f", rng.randrange(SLOTS), 128 * rng.randint(0, ROWS // 128)))
            forwards += 1
    return slot, SLOTS * slot + bf16.align(scratch), ops


def _forward(kind, st, slot, rows, bounded):
    kw = dict(T=T, K=K, D=D, F=F, num_layers=LAYERS, bounded=bounded)
    if kind == "bf16":
        got = bf16.plan_forward(st, rows, [rows], slot, scratch_only=False, **kw)
        return got["need"], got["fwd_state"]
    got = bs.plan_forward(st, rows, [rows], slot, storage=bs.MXFP8, **kw)
    return got["need"], got["offsets"]


def _forward_ranges(kind, rows, need, o):
    """(in the slot?, first byte, bytes) of what the launches of a forward write."""
    z, s = _sizes(kind, rows), bs.MXFP8
    kept = not need and o[4] >= 0
    if kind == "bf16":
        out = [(kept, o[1], z["xg"]), (kept, o[2], z["h1"]), (False, o[3], z["h2"])]
    else:
        out = [(kept, o[6], z["xg"]), (kept, o[2], z["h1"]), (kept, o[8], z["h2"]), (False, o[5], sum(bs.row_sizes(rows, D, s))),
               (False, o[7], sum(bs.row_sizes(rows, F, s)))]
    if need and o[0] >= 0:
        out.append((True, o[0], z["x"]))
    if kept:
        out.append((True, o[4], z["h3"]))
    return out


def _escapes(kind, seed, bounded):
    """Bytes outside their region: outside the arena, or a save outside its slot."""
    slot_bytes, arena, ops = _scenario(kind, seed)
    st = bf16.PlannerState(SLOTS, 1, slot_bytes, arena)
    held, arena_escapes, slot_escapes = [], 0, 0
    for op in ops:
        if op[0] == "f":
            need, o = _forward(kind, st, op[1], op[2], bounded)
            held.append((op[2], need, o))
            for inside, at, size in _forward_ranges(kind, op[2], need, o):
                arena_escapes += at < 0 or at + size > arena
                lo, hi = (op[1] * slot_bytes, (op[1] + 1) * slot_bytes) if inside else (SLOTS * slot_bytes, arena)
                slot_escapes += at < lo or at + size > hi
        else:
            rows, need, o = held[op[1]]
            z = _sizes(kind, rows)
            if kind == "bf16":
                b = bf16.plan_backward(st, rows, [rows], need, o, T=T, K=K, D=D, F=F)
                spans = list(zip(b, (z["xg"], z["h1"], z["h2"], z["h2"], z["xg"], z["h1"])))
            else:
                b = bs.plan_backward(st, rows, [rows], need, o, T=T, K=K, D=D, F=F, storage=bs.MXFP8)["offsets"]
                spans = [(b[7], z["xg"]), (b[1], z["h1"]), (b[9], z["h2"]), (b[11], z["xg"]), (b[3], bf16.align(rows * 2 * F))]
            arena_escapes += sum(at < 0 or at + size > arena for at, size in spans)
    return arena_escapes, slot_escapes


@pytest.mark.parametrize("kind", ["bf16", "mxfp8"])
def test_bounded_plans_stay_inside(kind):
    unbounded = [_escapes(kind, seed, False) for seed in range(60)]
    assert sum(a for a, _ in unbounded) > 0 and sum(s for _, s in unbounded) > 0  # why the launches use the bounded form
    assert [_escapes(kind, seed, True) for seed in range(60)] == [(0, 0)] * 60


def test_orderly_calls_are_planned_as_ever():
    for seed in range(20):
        slot_bytes, arena, _ = _scenario("bf16", seed)
        a, b = (bf16.PlannerState(SLOTS, 1, slot_bytes, arena) for _ in range(2))
        fa, fb = ([_forward("bf16", st, 1, 128 * (i + 1), bounded) for i in range(LAYERS)] for st, bounded in ((a, False), (b, True)))
        assert fa == fb and a.snapshot() == b.snapshot()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["bf16", "mxfp8"])
@pytest.mark.parametrize("seed", [0, 1, 2, 3, 4, 5])
def test_planner_kernels_match_the_oracle(kind, seed):
    import ctypes

    from dist_moe_b200 import _native as nat

    dev = torch.device("cuda", 0)
    i64 = lambda v: torch.tensor(v, dtype=torch.int64, device=dev)  # noqa: E731
    slot_bytes, arena, ops = _scenario(kind, seed)
    st = bf16.PlannerState(SLOTS, 1, slot_bytes, arena)
    offs, saved, peak, layer = i64(st.buffer_offsets), i64(st.saved), i64(st.peak), i64(st.layer)
    status = torch.zeros(8, dtype=torch.int32, device=dev)
    storage = (ctypes.c_int * 6)(*bs.MXFP8.as_list())
    held = []
    for op in ops:
        if op[0] == "f":
            want = _forward(kind, st, op[1], op[2], True)
            rows = torch.tensor([op[2]], dtype=torch.int32, device=dev)
            need, cond = torch.zeros(1, dtype=torch.uint8, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
            state, table, sel = torch.zeros(6 if kind == "bf16" else 10, dtype=torch.int64, device=dev), i64([0] * 18), i64([op[1]])
            if kind == "bf16":
                rc = nat.lib.dm_plan_fwd_bf16(rows.data_ptr(), rows.data_ptr(), saved.data_ptr(), offs.data_ptr(),
                                              peak.data_ptr(), need.data_ptr(), cond.data_ptr(), state.data_ptr(),
                                              sel.data_ptr(), layer.data_ptr(), 1, T, K, D, F, slot_bytes, SLOTS, LAYERS, BOUNDED,
                                              status.data_ptr(), nat.stream_ptr())
            else:
                rc = nat.lib.dm_plan_fwd_blockscaled(rows.data_ptr(), rows.data_ptr(), None, saved.data_ptr(), offs.data_ptr(),
                                                     peak.data_ptr(), need.data_ptr(), cond.data_ptr(), state.data_ptr(),
                                                     table.data_ptr(), sel.data_ptr(), layer.data_ptr(), 1, T, K, D, F,
                                                     storage, 1 << 20, slot_bytes, SLOTS, LAYERS, 0, 0, BOUNDED, 0, 0,
                                                     status.data_ptr(), nat.stream_ptr())
            nat.check(rc, "plan forward")
            assert (bool(need.item()), state.tolist()) == (want[0], want[1]) and cond.item() == int(want[0])
            held.append((rows, need, state, op[2], want))
        else:
            rows, need, state, n, want = held[op[1]]
            if kind == "bf16":
                b = bf16.plan_backward(st, n, [n], want[0], want[1], T=T, K=K, D=D, F=F)
                bo = i64([0] * 6)
                rc = nat.lib.dm_plan_bwd_bf16(rows.data_ptr(), rows.data_ptr(), saved.data_ptr(), offs.data_ptr(),
                                              peak.data_ptr(), need.data_ptr(), state.data_ptr(), bo.data_ptr(),
                                              layer.data_ptr(), 1, T, K, D, F, slot_bytes, SLOTS, status.data_ptr(),
                                              nat.stream_ptr())
            else:
                b = bs.plan_backward(st, n, [n], want[0], want[1], T=T, K=K, D=D, F=F, storage=bs.MXFP8)["offsets"]
                bo, bt = i64([0] * 16), i64([0] * 54)
                rc = nat.lib.dm_plan_bwd_blockscaled(rows.data_ptr(), rows.data_ptr(), saved.data_ptr(), offs.data_ptr(),
                                                     peak.data_ptr(), need.data_ptr(), state.data_ptr(), bo.data_ptr(),
                                                     bt.data_ptr(), layer.data_ptr(), 1, T, K, D, F, storage, 1 << 20,
                                                     slot_bytes, SLOTS, 0, 0, status.data_ptr(), nat.stream_ptr())
            nat.check(rc, "plan backward")
            assert bo.tolist() == b
        got = dict(buffer_offsets=offs.tolist(), saved=saved.tolist(), peak=peak.tolist(), layer=layer.tolist())
        assert got == st.snapshot(), op


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["bf16", "mxfp8"])
@pytest.mark.parametrize("factor,norm", [(None, False), (1.0, False), (1.0, True)])
def test_a_save_past_the_slot_does_not_run(fmt, factor, norm):
    """Slot 0 is driven past its end; slot 1 lies right behind it and keeps its bytes, outputs stay right, the backwards of the
    lost layers run, the status tells, and after a reset the context works as at first."""
    import dist_moe_b200 as dm

    dev = torch.device("cuda", 0)
    E, tokens = 4, 96
    g = torch.Generator().manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    w13 = (rnd(E, 2, 256, D) * D ** -0.5).bfloat16().to(dev).requires_grad_()
    w2 = (rnd(E, D, 256) * 256 ** -0.5).bfloat16().to(dev).requires_grad_()
    xs = [(rnd(tokens, D) * 0.5).bfloat16().to(dev).requires_grad_() for _ in range(4)]
    top = torch.topk(rnd(tokens, E), 2)
    ids, scores = top.indices.to(dev), torch.softmax(top.values, -1).to(dev).requires_grad_()
    post = dm.RMSNormPostprocess(eps=1e-6, norm_output_dtype=torch.float32, output_dtype=torch.bfloat16) if norm else None
    cfg = dm.Config(max_num_local_input_tokens=tokens, hidden_dim=D, intermediate_dim=256, top_k=2, num_experts=E,
                    max_moe_layers_per_activation_slot=2, num_activation_slots=2, activation_slot_capacity_factor=factor,
                    block_scaled=dm.BlockScaledConfig() if fmt == "mxfp8" else None)
    ctx = dm.create_context(group=None, config=cfg, device=dev)
    options = dm.ExecutionOptions(experts_output_postprocess=post)
    try:
        def run(x):
            return dm.routed_experts(x, ids, scores, w13, w2, ctx, options=options)

        def grads(out, x):
            return torch.autograd.grad(out, (x, scores, w13, w2), torch.ones_like(out))

        want = []
        for x in xs:
            out = run(x)
            want.append((out.detach(), grads(out, x)))
        ctx.check_status()
        state, size = ctx._state, ctx.memory_plan.activation_slot_bytes
        ctx.select_activation_slot(1, 2)
        outs = [run(xs[0])]  # slot 1 in use
        torch.cuda.synchronize()
        before = state.arena[size:2 * size].clone()
        ctx.select_activation_slot(0, 2)
        first, second = run(xs[0]), run(xs[1])
        grads(first, xs[0])  # out of order: the slot's free pointer stays ahead of what is counted
        grads(second, xs[1])
        outs += [run(x) for x in xs]  # and two layers more than the slot was made for
        torch.cuda.synchronize()
        assert torch.equal(state.arena[size:2 * size], before)
        for out, (w, _) in zip(outs[1:], want):
            assert torch.equal(out, w)
        for out, x in reversed(list(zip(outs[1:], xs))):
            grads(out, x)
        with pytest.raises(RuntimeError, match="arena overflow"):
            ctx.check_status()
        got = grads(outs[0], xs[0])  # slot 1 was left alone
        for a, b in zip(got, want[0][1]):
            assert torch.equal(a, b)
        ctx.reset()
        out = run(xs[2])
        assert torch.equal(out, want[2][0])
        for a, b in zip(grads(out, xs[2]), want[2][1]):
            assert torch.equal(a, b)
        ctx.check_status()
    finally:
        ctx.close()
