"""SwiGLU epilogue of the BF16 forward GEMM on tiles that end inside a 32-row block, around the steps of four rows that it
works in: the bits of the SwiGLU kernel on the same h1."""

import pytest
import torch

from tests.test_gemm_gpu import _native

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
COUNTS = [[1, 2, 3, 4, 5, 0, 7, 8, 9], [12, 13, 15, 16, 17], [20, 21, 31, 32, 33, 36, 37]]


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("clamped", [0, 1])
def test_bf16_few_rows(counts, clamped):
    nat = _native()
    gen = torch.Generator(device=DEV).manual_seed(31)
    R, K, F = sum(counts), 128, 256
    x = torch.randn(R, K, device=DEV, generator=gen).bfloat16()
    w = torch.randn(len(counts), 2 * F, K, device=DEV, generator=gen).bfloat16()
    offs = torch.tensor([0] + counts, device=DEV).cumsum(0).int()
    arena = torch.zeros((R + 300) * K * 2, dtype=torch.uint8, device=DEV)
    arena[: R * K * 2] = x.view(torch.uint8).reshape(-1)
    h1, h2, want = (torch.full((R + 1, n), 5.0, device=DEV, dtype=torch.bfloat16) for n in (2 * F, F, F))
    status = torch.zeros(8, dtype=torch.int32, device=DEV)
    op = lambda t: nat.Operand(t.data_ptr(), t.numel() * t.element_size(), None)  # noqa: E731
    nat.check(nat.lib.dm_gemm_fprop(op(arena), w.data_ptr(), op(h1), op(h2), None, offs.data_ptr(), len(counts), R, 2 * F, K,
                                    1, clamped, 1.702, 7.0, None, 0, status.data_ptr(), nat.stream_ptr()), "fprop")
    rows = torch.tensor([R], dtype=torch.int32, device=DEV)
    nat.check(nat.lib.dm_swiglu_fwd(h1.data_ptr(), None, want.data_ptr(), None, rows.data_ptr(), R, F, clamped, 1.702, 7.0,
                                    None, 0.0, None, nat.stream_ptr()), "dm_swiglu_fwd")
    torch.cuda.synchronize()
    assert status[0].item() == 0, status.tolist()
    assert torch.equal(h2, want) and bool((h2[R] == 5.0).all()) and bool(torch.isfinite(h1).all())
