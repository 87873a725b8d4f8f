"""Pairs left out of launches whose last round would use a part of them: the bits of the launch that gives every tile a pair of its
own, at tiles of the rows where the rule begins and ends, with rounds that come out even, short by one tile and far from full."""

import pytest
import torch

from tests.test_gemm_blockscaled_rows_gpu import _Launch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", _Launch.FORMS)
@pytest.mark.parametrize("counts", [[32, 7, 0, 31, 1], [33, 7, 0, 31, 1]], ids=["32 rows", "33 rows"])
def test_mxfp8(form, counts):
    one_each = _Launch(form, counts, 256, 768, 0).run(0)  # 12 tiles
    launch = _Launch(form, counts, 256, 768, 0)
    for num_sms in (8, 10, 14, 16, 22):
        for a, b in zip(one_each, launch.run(num_sms)):
            assert torch.equal(a, b), num_sms


@pytest.mark.parametrize("counts", [[128, 3, 0, 90], [130, 3, 0, 90], [256, 1, 20, 0]])
@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("dispatch", [False, True])
def test_bf16(counts, backward, dispatch):
    from dist_moe_b200 import _native as nat

    dev, n, kd, e, rows = torch.device("cuda", 0), 1280, 192, len(counts), sum(counts)
    torch.manual_seed(rows + backward)
    offs = torch.tensor([sum(counts[:i]) for i in range(e + 1)], dtype=torch.int32, device=dev)
    x = torch.randn(rows + 300, kd, device=dev).bfloat16()
    w = (torch.randn(e, kd, n, device=dev) if backward else torch.randn(e, n, kd, device=dev)).mul_(0.1).bfloat16()
    ptrs = x.data_ptr() + torch.arange(rows, device=dev) * kd * 2
    flags = torch.zeros(rows // 128 + 2, dtype=torch.int32, device=dev)
    status = torch.zeros(8, dtype=torch.int32, device=dev)
    op = lambda t: nat.Operand(t.data_ptr(), t.numel() * 2, None)  # noqa: E731
    none = nat.Operand(None, 0, None)

    def run(num_sms):
        out = torch.full((rows + 8, n), 5.0, device=dev, dtype=torch.bfloat16)
        pulled = torch.full((rows + 300, kd), float("nan"), device=dev, dtype=torch.bfloat16)
        head = (ptrs.data_ptr(), flags.data_ptr(), op(pulled)) if dispatch else (op(x),)
        table = (offs.data_ptr(), e, rows, n, kd)
        end = (None, num_sms, status.data_ptr(), nat.stream_ptr())
        if backward:
            fn = nat.lib.dm_gemm_dgrad_dispatch if dispatch else nat.lib.dm_gemm_dgrad
            rc = fn(*head, w.data_ptr(), op(out), *(() if dispatch else (None,)), *table, *end)
        else:
            fn = nat.lib.dm_gemm_fprop_dispatch if dispatch else nat.lib.dm_gemm_fprop
            rc = fn(*head, w.data_ptr(), op(out), none, *(() if dispatch else (None,)), *table, 0, 0, 1.0, 0.0, *end)
        nat.check(rc, "gemm")
        torch.cuda.synchronize()
        assert status[0].item() == 0, status.tolist()
        return out.view(torch.int16)

    want = run(0)
    assert bool((want[:rows] != want[rows]).any(dim=1).all()), "every row is written"
    for num_sms in (4, 8, 14, 16, 28):
        assert torch.equal(run(num_sms), want), num_sms
