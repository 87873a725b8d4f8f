"""Fused dispatch with gather units of 1, 2, 4 and 8 rows: at the row counts where the unit changes (24 gather warps for six SMs), with
rows that fill the 16-byte loads of a warp once, several times and in part, null pointers, and a ragged last unit.  The gathered copy
is exact, and the product equals that of the same rows without a dispatch bit for bit (the same tiles in the same order)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
SMS = 6
WARPS = 4 * SMS


@pytest.mark.parametrize("rows", [1, WARPS, WARPS + 1, 2 * WARPS + 1, 4 * WARPS, 4 * WARPS + 1, 333])
@pytest.mark.parametrize("kd", [64, 1024, 1088, 2112])  # 8, 128 (four rows at a time), 136 and 264 (two) pieces of 16 bytes
def test_units_of_every_size(rows, kd):
    from dist_moe_b200 import _native as nat

    dev, n = torch.device("cuda", 0), 256
    torch.manual_seed(rows + kd)
    cut = rows // 3
    offs = torch.tensor([0, cut, cut, rows], dtype=torch.int32, device=dev)
    src = torch.randn(rows + 3, kd, device=dev).bfloat16()
    index = torch.randint(0, rows + 3, (rows,), device=dev)
    ptrs = src.data_ptr() + index.to(torch.int64) * kd * 2
    want = src[index].clone()
    ptrs[rows // 2] = 0
    want[rows // 2] = 0
    w = (torch.randn(3, n, kd, device=dev) * 0.1).bfloat16()
    flags = torch.full((rows // 128 + 8,), 77, dtype=torch.int32, device=dev)
    status = torch.zeros(8, dtype=torch.int32, device=dev)
    op = lambda t: nat.Operand(t.data_ptr(), t.numel() * 2, None)  # noqa: E731
    none = nat.Operand(None, 0, None)
    got_a = torch.full((rows + 300, kd), 9.0, device=dev, dtype=torch.bfloat16)
    plain_a = torch.zeros(rows + 300, kd, device=dev, dtype=torch.bfloat16)
    plain_a[:rows] = want
    got, plain = (torch.zeros(rows, n, device=dev, dtype=torch.bfloat16) for _ in range(2))
    tail = (offs.data_ptr(), 3, rows, n, kd, 0, 0, 1.0, 0.0, None, SMS, status.data_ptr(), nat.stream_ptr())
    nat.check(nat.lib.dm_gemm_fprop_dispatch(ptrs.data_ptr(), flags.data_ptr(), op(got_a), w.data_ptr(), op(got), none, *tail), "dispatch")
    nat.check(nat.lib.dm_gemm_fprop(op(plain_a), w.data_ptr(), op(plain), none, None, *tail), "plain")
    torch.cuda.synchronize()
    assert status[0].item() == 0, status.tolist()
    assert torch.equal(got_a[:rows].view(torch.int16), want.view(torch.int16))
    assert bool((got_a[rows:] == 9.0).all()), "nothing past the last row is written"
    assert torch.equal(got.view(torch.int16), plain.view(torch.int16))
