"""Where a weight gradient goes: a GEMM writes every expert's part, so a parameter of another size is refused before anything is
allocated or launched, also for MXFP8, whose source weights are not looked at after the forward (CPU)."""

import types

import pytest
import torch

from dist_moe_b200 import _bf16
from dist_moe_b200._execution import ExecutionOptions

SHAPE = (4, 6, 8)
CONFIG = types.SimpleNamespace(wgrad_dtype=None)


def _destination(param, explicit=None, **options):
    return _bf16._wgrad_destination(param, SHAPE, ExecutionOptions(**options), CONFIG, None, explicit)


@pytest.mark.parametrize("shape", [(2, 6, 8), (5, 6, 8), (4, 2, 3, 4)])
@pytest.mark.parametrize("how", ["fresh", "dtype", "tensor", "accumulate"])
def test_another_size_is_refused(shape, how):
    param = torch.zeros(shape, dtype=torch.bfloat16)
    explicit = {"dtype": torch.float32, "tensor": torch.zeros(shape)}.get(how)
    with pytest.raises(RuntimeError):
        _destination(param, explicit, inplace_wgrad_accum=how == "accumulate")
    assert param.grad is None


@pytest.mark.parametrize("shape", [(4, 6, 8), (4, 2, 3, 8), (24, 8)])
def test_the_same_size_in_any_shape(shape):
    param = torch.zeros(shape, dtype=torch.bfloat16)
    dst, accumulate, returned = _destination(param)
    assert dst.shape == param.shape and dst.is_contiguous() and (accumulate, returned) == (0, True)
    assert _destination(param, torch.float32)[0].dtype is torch.float32
    own = torch.zeros(shape)
    assert _destination(param, own)[0] is own
    assert _destination(param, inplace_wgrad_accum=True)[0] is param.grad
