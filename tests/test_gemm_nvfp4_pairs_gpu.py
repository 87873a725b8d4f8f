"""NVFP4 GEMM on CTA pairs (256 x 256 tiles) at the edges of its tiles, against the 128 x 256 kernel: both accumulate the same K
steps in the same order and round at the same places, so the rows that are written are equal bit for bit; and against the fp32
product of the dequantised operands."""

import pytest
import torch

from tests.test_gemm_blockscaled_gpu import _close, _nat
from tests.test_gemm_blockscaled_swapped_gpu import _operands

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# no row, one row, one more than a CTA's 128 and than a tile's 256, tiles whose odd CTA has no rows
COUNTS = [[1, 0, 129, 256, 257], [31, 384], [0, 0], [1040]]


def _run(nat, pairs, a, sa, qw, sw, c, h2, ptrs, inv, einv, offs, cnts, E, R, N, K, swiglu):
    status = torch.zeros(8, dtype=torch.int32, device=DEV)
    none = nat.Operand(None, 0, None)
    op = lambda t: none if t is None else nat.Operand(t.data_ptr(), t.numel() * t.element_size(), None)  # noqa: E731
    head = (op(a), sa, qw.data_ptr(), sw.data_ptr(), op(c), op(h2), nat.ptr(ptrs), op(inv), nat.ptr(einv), offs.data_ptr())
    tail = (E, R, N, K, swiglu, 0, 1.702, 7.0, None, 0, status.data_ptr(), nat.stream_ptr())
    if pairs:
        nat.check(nat.lib.dm_gemm_nvfp4_pairs(*head, cnts.data_ptr(), *tail), "pairs")
    else:
        nat.check(nat.lib.dm_gemm_blockscaled(1, *head, *tail), "wide")
    torch.cuda.synchronize()
    return status.cpu()


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("K,N", [(256, 384), (1536, 256)])
def test_dense_and_scattered_rows(counts, K, N):
    nat = _nat()
    E, off, real, R, (qa, sa, da, inv), (qw, sw, dw, einv), offs, cnts = _operands(nat, 1, counts, K, N, 5 + K)
    scales = nat.Operand(sa.data_ptr(), sa.numel() * sa.element_size(), None)
    # the rows' scales again, 48 bytes into their buffer and named by a device offset
    shifted = torch.zeros(sa.numel() * sa.element_size() + 256, dtype=torch.uint8, device=DEV)
    shifted[48:48 + sa.numel() * sa.element_size()] = sa.view(torch.uint8).reshape(-1)
    where = torch.tensor([48], dtype=torch.int64, device=DEV)
    moved = nat.Operand(shifted.data_ptr(), shifted.numel(), where.data_ptr())
    want, got, again = (torch.full((R + 8, N), 5.0, device=DEV, dtype=torch.bfloat16) for _ in range(3))
    rest = (qw, sw)
    for pairs, sf, dst in ((False, scales, want), (True, scales, got), (True, moved, again)):
        status = _run(nat, pairs, qa, sf, *rest, dst, None, None, inv, einv, offs, cnts, E, R, N, K, 0)
        assert status[0].item() == 0, status.tolist()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(again.view(torch.int16), want.view(torch.int16))
    for e, n in enumerate(counts):
        rows = torch.arange(off[e], off[e] + n)
        if n:
            _close(got.cpu()[rows], da[rows] @ dw[e].T, f"expert {e}")
    sct = torch.full((R, N), 5.0, device=DEV, dtype=torch.bfloat16)
    perm = torch.randperm(R, device=DEV)
    ptrs = torch.zeros(R, dtype=torch.int64, device=DEV)
    ptrs[real.to(DEV)] = sct.data_ptr() + perm[real.to(DEV)].to(torch.int64) * (N * 2)
    _run(nat, True, qa, scales, *rest, None, None, ptrs, inv, einv, offs, cnts, E, R, N, K, 0)
    index = perm[real.to(DEV)]
    assert torch.equal(sct[index].view(torch.int16), want[real.to(DEV)].view(torch.int16))
    untouched = torch.ones(R, dtype=torch.bool, device=DEV)
    untouched[index] = False
    assert bool((sct[untouched] == 5.0).all())


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("with_h1", [False, True])
def test_swiglu_rows(counts, with_h1):
    """At 2F = 384 the last tile's upper 128 columns do not exist."""
    nat, K, F = _nat(), 512, 192
    E, off, real, R, (qa, sa, da, inv), (qw, sw, dw, einv), offs, cnts = _operands(nat, 1, counts, K, 2 * F, 9, F)
    scales = nat.Operand(sa.data_ptr(), sa.numel() * sa.element_size(), None)
    out = {}
    for pairs in (False, True):
        h1 = torch.full((R, 2 * F), 5.0, device=DEV, dtype=torch.bfloat16) if with_h1 else None
        h2 = torch.full((R, F), 5.0, device=DEV, dtype=torch.bfloat16)
        status = _run(nat, pairs, qa, scales, qw, sw, h1, h2, None, inv, einv, offs, cnts, E, R, 2 * F, K, 1)
        assert status[0].item() == 0, status.tolist()
        out[pairs] = (h1, h2)
    live = torch.zeros(R, dtype=torch.bool, device=DEV)
    live[real.to(DEV)] = True
    for want, got in zip(out[False], out[True]):
        if got is not None:
            assert torch.equal(got[live].view(torch.int16), want[live].view(torch.int16))
            assert bool((got[~live] == 5.0).all()), "rows past the count are left alone"


def test_groups_that_are_not_padded_are_left_out():
    nat, K, N = _nat(), 256, 128
    E, off, real, R, (qa, sa, da, inv), (qw, sw, dw, einv), _, _ = _operands(nat, 1, [128, 128], K, N, 3)
    offs = torch.tensor([0, 32, 160], dtype=torch.int32, device=DEV)
    cnts = torch.tensor([32, 128], dtype=torch.int32, device=DEV)
    scales = nat.Operand(sa.data_ptr(), sa.numel() * sa.element_size(), None)
    out = torch.full((R, N), 5.0, device=DEV, dtype=torch.bfloat16)
    status = _run(nat, True, qa, scales, qw, sw, out, None, None, inv, einv, offs, cnts, E, R, N, K, 0)
    assert status[0].item() != 0
    assert bool((out[32:] == 5.0).all())
