"""SwiGLU at every bf16 gate: the branch-free reciprocal inside the sigmoid gives the bits of the IEEE one."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("clamped,alpha,limit", [(0, 1.0, 0.0), (1, 1.702, 7.0), (1, 30.0, 3.0e38)])
def test_every_gate(clamped, alpha, limit):
    """All 65 536 bit patterns (tiny sigmoids, infinities and NaNs among them), eight to a thread in shuffled order, against
    the same fp32 expression with torch's exponential and division; alpha 30 drives the reciprocal into subnormals."""
    from dist_moe_b200 import _native as nat

    gates = torch.arange(65536, dtype=torch.int32, device=DEV).to(torch.int16).view(torch.bfloat16)
    gates = gates[torch.randperm(65536, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5))]
    R, F = 64, 1024
    ups = torch.randn(R, F, device=DEV, generator=torch.Generator(device=DEV).manual_seed(6)).bfloat16()
    h1 = torch.cat([gates.view(R, F), ups], 1).contiguous()
    h2 = torch.empty(R, F, dtype=torch.bfloat16, device=DEV)
    rows = torch.tensor([R], dtype=torch.int32, device=DEV)
    nat.check(nat.lib.dm_swiglu_fwd(h1.data_ptr(), None, h2.data_ptr(), None, rows.data_ptr(), R, F, clamped, alpha, limit,
                                    None, 0.0, None, nat.stream_ptr()), "dm_swiglu_fwd")
    g, u = gates.view(R, F).float(), ups.float()
    if clamped:
        g = torch.fmin(g, torch.tensor(limit, device=DEV))  # as fminf: a NaN gate becomes the limit
        z = g * (1.0 / (1.0 + torch.exp(-(alpha * g)))) * (u.clamp(-limit, limit) + 1.0)
    else:
        z = g * (1.0 / (1.0 + torch.exp(-g))) * u
    want = z.bfloat16()
    both_nan = torch.isnan(want) & torch.isnan(h2)
    assert torch.equal(h2.view(torch.int16)[~both_nan], want.view(torch.int16)[~both_nan])
