"""Fused dispatch that finds its flags clear and leaves them clear: launches of changing sizes one after another on one scratch, also
with no rows and with a predicate that is off, give what launches with a scratch cleared by the call give."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sms", [0, 2, 6])
@pytest.mark.parametrize("backward", [False, True])
def test_flags_stay_clear_from_launch_to_launch(sms, backward):
    from dist_moe_b200 import _native as nat

    dev, n, kd, experts = torch.device("cuda", 0), 256, 320, 3
    torch.manual_seed(sms + backward)
    kept = torch.zeros(3000 // 128 + 3, dtype=torch.int32, device=dev)
    dirty = torch.full((3000 // 128 + 3,), 77, dtype=torch.int32, device=dev)
    status = torch.zeros(8, dtype=torch.int32, device=dev)
    w = (torch.randn(experts, kd if backward else n, n if backward else kd, device=dev) * 0.1).bfloat16()
    op = lambda t: nat.Operand(t.data_ptr(), t.numel() * 2, None)  # noqa: E731
    none = nat.Operand(None, 0, None)
    # live rows, max_rows, predicate: the ticket's place and the number of flags change; fewer live rows than max_rows, and none
    for rows, max_rows, on in [(1, 1, 1), (128, 128, 1), (129, 3000, 1), (3000, 3000, 1), (0, 200, 1), (700, 700, 0), (700, 701, 1),
                               (700, 701, 1)]:
        offs = torch.tensor([0, rows // 3, rows // 3, rows], dtype=torch.int32, device=dev)
        src = torch.randn(max_rows, kd, device=dev).bfloat16()
        ptrs = src.data_ptr() + torch.randint(0, max_rows, (max_rows,), device=dev) * kd * 2
        cond = torch.tensor([on], dtype=torch.int32, device=dev)
        outs = []
        for flags, extra in ((kept, nat.GATHER_FLAGS_KEPT_CLEAR), (dirty, 0)):
            a = torch.full((max_rows + 300, kd), 9.0, device=dev, dtype=torch.bfloat16)
            c = torch.full((max_rows, n), 5.0, device=dev, dtype=torch.bfloat16)
            end = (cond.data_ptr(), sms | extra, status.data_ptr(), nat.stream_ptr())
            head = (ptrs.data_ptr(), flags.data_ptr(), op(a), w.data_ptr(), op(c))
            if backward:
                rc = nat.lib.dm_gemm_dgrad_dispatch(*head, offs.data_ptr(), experts, max_rows, n, kd, *end)
            else:
                rc = nat.lib.dm_gemm_fprop_dispatch(*head, none, offs.data_ptr(), experts, max_rows, n, kd, 0, 0, 1.0, 0.0, *end)
            nat.check(rc, "dispatch")
            outs.append((a, c))
        torch.cuda.synchronize()
        assert status[0].item() == 0, status.tolist()
        assert not kept.any().item(), (rows, max_rows, kept.tolist())
        for left, right in zip(*outs):
            assert torch.equal(left.view(torch.int16), right.view(torch.int16)), (rows, max_rows)
        assert bool((outs[0][1][:rows] != 5.0).any()) == (on == 1 and rows > 0)
