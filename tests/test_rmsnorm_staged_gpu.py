"""RMSNorm + weighted sum forward with a token's rows staged in shared memory, against the form that reads them from memory: the
same sums in the same order, so equal bit for bit.  The second form is reached with more rows per token than the first takes
(K = 32 at D > 3456); rows past the first are given ids of -1, which are left out of sum and result."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _nat():
    from dist_moe_b200 import _native

    return _native


def _run(h3, scores, ids, gamma, norm_bf16, kahan, save):
    nat = _nat()
    T, K, D = h3.shape
    out = torch.full((T, D), 7.0, dtype=torch.bfloat16, device=DEV)
    rstd = torch.full((T, K), 7.0, device=DEV)
    kept = torch.full_like(h3, 3.0) if save else None
    nat.check(nat.lib.dm_rmsnorm_combine_fwd(
        h3.data_ptr(), scores.data_ptr(), int(scores.dtype is torch.bfloat16), ids.data_ptr(), int(ids.dtype is torch.int64),
        nat.ptr(gamma), 0.25, 1e-6, int(norm_bf16), int(kahan), out.data_ptr(), rstd.data_ptr(), T, K, D, nat.ptr(kept), None, None,
        0, nat.stream_ptr()), "dm_rmsnorm_combine_fwd")
    torch.cuda.synchronize()
    return out, rstd, kept


@pytest.mark.parametrize("T", [1, 700, 2500])  # fewer tokens than blocks, one and several rounds
@pytest.mark.parametrize("K,D,ids_dtype,score_dtype,with_gamma,norm_bf16,kahan", [
    (1, 3464, torch.int32, torch.float32, False, False, False), (3, 4104, torch.int64, torch.bfloat16, True, True, False),
    (4, 3464, torch.int64, torch.float32, True, False, True), (5, 4096, torch.int32, torch.bfloat16, False, True, True),
    (8, 6904, torch.int64, torch.float32, False, False, False), (7, 7680, torch.int64, torch.float32, False, True, False)])
def test_staged_rows_match_rows_in_memory(T, K, D, ids_dtype, score_dtype, with_gamma, norm_bf16, kahan):
    g = torch.Generator().manual_seed(T + K)
    wide = torch.randn(T, 32, D, generator=g).bfloat16().to(DEV) if T < 1000 else torch.randn(T, 32, D, device=DEV).bfloat16()
    scores = torch.rand(T, 32, generator=g).to(score_dtype).to(DEV)
    ids = torch.randint(0, 4, (T, 32), generator=g).to(ids_dtype).to(DEV)
    ids[:, K:] = -1
    ids[::7, 0] = -1  # routes that are left out
    gamma = torch.randn(D, generator=g).bfloat16().to(DEV) if with_gamma else None
    assert K * D * 2 <= 216 * 1024 < 32 * D * 2  # one form each
    want, want_rstd, _ = _run(wide, scores, ids, gamma, norm_bf16, kahan, False)
    own = [t[:, :K].contiguous() for t in (wide, scores, ids)]
    got, got_rstd, kept = _run(*own, gamma, norm_bf16, kahan, True)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(got_rstd, want_rstd[:, :K])
    assert torch.equal(kept, own[0])


def test_smallest_rows():
    """D = 8: one vector per row, against float64."""
    T, K, D = 5, 4, 8
    g = torch.Generator().manual_seed(1)
    h3 = torch.randn(T, K, D, generator=g).bfloat16()
    scores, ids = torch.rand(T, K, generator=g), torch.zeros(T, K, dtype=torch.int32)
    got, rstd, _ = _run(h3.to(DEV), scores.to(DEV), ids.to(DEV), None, False, False, False)
    x = h3.double()
    r = torch.rsqrt(x.pow(2).mean(-1) + 1e-6)
    want = (x * r[..., None] * scores.double()[..., None]).sum(1)
    assert torch.allclose(rstd.cpu().double(), r, rtol=1e-5)  # fp32 sum of eight squares and rsqrtf
    assert bool(((got.cpu().double() - want).abs() <= want.abs() * 2 ** -8 + 1e-5).all())  # one bf16 rounding of an fp32 sum


@pytest.mark.parametrize("K,D", [(4, 6784), (4, 6792), (4, 6912), (4, 6920), (7, 3944)])
def test_where_the_number_of_buffers_changes(K, D):
    test_staged_rows_match_rows_in_memory(1500, K, D, torch.int64, torch.float32, False, False, False)


@pytest.mark.parametrize("T", [1, 2500])
@pytest.mark.parametrize("D", [8, 2048, 2056])
def test_a_single_row(T, D):
    """One row: read from memory up to D = 2048, staged beyond; 32 of them, all but one left out, are staged."""
    g = torch.Generator().manual_seed(T + D)
    wide, scores = torch.randn(T, 32, D, generator=g).bfloat16().to(DEV), torch.rand(T, 32, generator=g).to(DEV)
    ids = torch.full((T, 32), -1, dtype=torch.int64, device=DEV)
    ids[1:, 0] = 0
    want, want_rstd, _ = _run(wide, scores, ids, None, False, False, False)
    own = [t[:, :1].contiguous() for t in (wide, scores, ids)]
    got, got_rstd, kept = _run(*own, None, False, False, True)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(got_rstd, want_rstd[:, :1]) and torch.equal(kept, own[0])
