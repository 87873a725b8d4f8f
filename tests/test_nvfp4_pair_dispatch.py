"""Which NVFP4 products of a layer run on CTA pairs, and that it changes nothing but the time."""

import itertools

import pytest
import torch

from dist_moe_b200 import _blockscaled as bs

# experts, hidden, intermediate, SwiGLU in the epilogue, rows per expert, us of W13 on 128 x 256 tiles | pairs, of W2 likewise (one B200)
MEASURED = [
    (32, 7168, 2048, True, 512, 239, 231, 165, 178), (32, 7168, 2048, True, 2048, 807, 745, 565, 569),
    (8, 2048, 768, True, 512, 21.9, 19.7, 12.9, 19.4), (8, 2048, 768, True, 2048, 57, 47, 35, 43),
    (32, 2048, 768, True, 512, 61, 55, 39, 49), (32, 2048, 768, True, 1024, 100, 84, 62, 81),
    (16, 4096, 1024, True, 1024, 84, 73, 64, 81), (16, 4096, 1024, True, 2048, 143, 126, 112, 147),
    (32, 4096, 1536, True, 512, 125, 114, 83, 97), (32, 4096, 1536, True, 2048, 391, 356, 274, 305),
    (16, 7168, 768, True, 512, 57.4, 61.1, 54, 75), (16, 7168, 768, True, 768, 83, 73, 74, 105),
    (8, 7168, 1024, True, 512, 41.2, 48.4, 34, 44), (8, 7168, 1024, True, 768, 53, 49, 45, 59), (8, 7168, 1024, True, 2048, 115, 103, 97, 129),
    (32, 5120, 1280, True, 512, 124, 116, 93, 109), (32, 5120, 1280, True, 2048, 388, 350, 311, 356),
    (8, 1536, 4096, True, 512, 64, 60, 26.7, 24.6), (8, 2048, 4096, True, 512, 69, 64, 27.6, 31.7), (8, 2048, 4096, True, 2048, 209, 182, 78, 66),
    (4, 4096, 7168, True, 768, 102, 94, 53, 51.5), (4, 4096, 7168, True, 2048, 226, 204, 118, 98), (16, 1280, 3584, True, 2048, 329, 293, 84, 75),
    (16, 7168, 2048, False, 512, 138, 120, 86, 92), (16, 7168, 2048, False, 2048, 443, 368, 282, 290),
    (16, 4096, 1024, False, 2048, 148, 124, 110, 148), (16, 2048, 768, False, 512, 27.3, 32.5, 21.4, 30.7),
    (16, 2304, 1024, False, 512, 36.4, 40.4, 27.8, 32.3), (16, 2304, 1024, False, 2048, 103, 94, 68, 88),
]


@pytest.mark.parametrize("case", MEASURED, ids=lambda c: "x".join(map(str, c[:5])))
def test_the_rule_takes_the_faster_kernel(case):
    E, D, F, fused, rows, *times = case
    for n, kd, swiglu, (wide, pairs) in ((2 * F, D, fused, times[:2]), (D, F, False, times[2:])):
        assert bs._on_pairs(E * rows, E, n, kd, swiglu, 0) == (pairs < wide), (n, kd)


def test_few_rows_stay_where_they_are():
    for E, D, F in ((8, 2048, 768), (32, 7168, 2048), (4, 7168, 7168)):
        for rows in (0, 1, 511):
            assert not bs._on_pairs(E * rows, E, 2 * F, D, True, 0) and not bs._on_pairs(E * rows, E, D, F, False, 0)


def _layer(T, D, F, K, E, fuse, seed=3):
    import dist_moe_b200 as dm

    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(T, D, generator=g) * 0.1).bfloat16().to(dev)
    w13, w2 = (torch.randn(E, 2, F, D, generator=g) * D**-0.5).bfloat16().to(dev), (torch.randn(E, D, F, generator=g) * F**-0.5).bfloat16().to(dev)
    logits = torch.randn(T, E, generator=g)
    logits[:, 0] += 1.5  # one expert with many tiles of rows, the last one without any
    logits[:, -1] = -100.0
    top = torch.topk(torch.softmax(logits, -1), K)
    ids = torch.where(torch.rand(T, K, generator=g) < 0.05, -1, top.indices).to(dev)
    cfg = dm.Config(max_num_local_input_tokens=T, hidden_dim=D, intermediate_dim=F, top_k=K, num_experts=E,
                    max_moe_layers_per_activation_slot=1, inference=True, num_activation_slots=0,
                    block_scaled=dm.BlockScaledConfig(format=dm.BlockScaledFormat.NVFP4))
    ctx = dm.create_context(group=None, config=cfg, device=dev)
    weights = (dm.prepare_block_scaled_weight(w13, cfg, fuse_swiglu=fuse, inference=True), dm.prepare_block_scaled_weight(w2, cfg, inference=True))
    return ctx, lambda: dm.routed_experts(x, ids, top.values.float().to(dev), *weights, ctx)


@pytest.mark.gpu
@pytest.mark.parametrize("fuse", [True, False])
@pytest.mark.parametrize("T,D,F,K,E", [(300, 512, 256, 2, 4), (1111, 256, 768, 3, 6)])
def test_a_layer_on_pairs_gives_the_same_bits(fuse, T, D, F, K, E, monkeypatch):
    """Either product on either kernel, over a workspace that holds NaN of every kind before the call."""
    monkeypatch.setattr(bs, "SWAPPED_MAX_ROWS_PER_EXPERT", 0)
    ctx, call = _layer(T, D, F, K, E, fuse)
    try:
        outs = []
        for pairs13, pairs2 in itertools.product((False, True), repeat=2):
            monkeypatch.setattr(bs, "_on_pairs", lambda routes, experts, n, kd, swiglu, sms: pairs13 if n == 2 * F and kd == D else pairs2)
            bs._workspace(ctx._state)[1].fill_(255)
            outs.append(call())
            ctx.check_status()
        assert torch.isfinite(outs[0]).all() and bool((outs[0] != 0).any())
        for out in outs[1:]:
            assert torch.equal(out.view(torch.int16), outs[0].view(torch.int16))
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [511, 512])
def test_a_call_at_the_line(rows, monkeypatch):
    """The rule as it is, at 512 rows per expert and one route in eight below it."""
    import dist_moe_b200._native as nat

    used = []
    monkeypatch.setattr(bs, "_gemm_pairs", lambda f, *a: used.append(a) or nat.lib.dm_gemm_nvfp4_pairs(*a))
    T, D, F, K, E = rows, 512, 2304, 4, 4
    ctx, call = _layer(T, D, F, K, E, True)
    try:
        out = call()
        ctx.check_status()
        assert len(used) == (0 if rows < 512 else sum(bs._on_pairs(T * K, E, n, kd, s, 0) for n, kd, s in ((2 * F, D, True), (D, F, False))))
        assert (rows < 512) == (len(used) == 0)
        monkeypatch.setattr(bs, "_on_pairs", lambda *a: False)
        assert torch.equal(call().view(torch.int16), out.view(torch.int16))
    finally:
        ctx.close()
