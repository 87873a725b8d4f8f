"""The branch-free reciprocal of the sigmoid against CUDA's IEEE reciprocal, bit for bit, over every float of its range."""

import ctypes
import subprocess
from pathlib import Path

import pytest
import torch

from dist_moe_b200 import build

pytestmark = pytest.mark.gpu
CSRC = Path(__file__).resolve().parents[1] / "dist_moe_b200" / "csrc"

SOURCE = r"""
#include "common.cuh"

// Floats with bit patterns [first, first + count): how many reciprocals differ, and one of them.
__global__ void differ(uint32_t first, uint32_t count, unsigned long long* n, uint32_t* which) {
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const float d = __uint_as_float(first + static_cast<uint32_t>(i));
    if (__float_as_uint(dm::rcp_newton(d)) != __float_as_uint(__frcp_rn(d))) {
      atomicAdd(n, 1ull);
      *which = first + static_cast<uint32_t>(i);
    }
  }
}

extern "C" int check(uint32_t first, uint32_t count, unsigned long long* n, uint32_t* which, void* stream) {
  differ<<<1184, 256, 0, static_cast<cudaStream_t>(stream)>>>(first, count, n, which);
  return static_cast<int>(cudaGetLastError());
}
"""


def test_every_float_from_one_to_two_to_the_126(tmp_path):
    (tmp_path / "check.cu").write_text(SOURCE)
    subprocess.run([build.find_nvcc(), *build.NVCC_FLAGS, "-shared", f"-I{CSRC}", "-o", str(tmp_path / "check.so"),
                    str(tmp_path / "check.cu")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "check.so"))
    lib.check.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    found = torch.zeros(2, dtype=torch.int64, device="cuda:0")
    first, last = 0x3F800000, 0x7E800000  # 1 and 2^126
    at = first
    while at <= last:
        count = min(1 << 28, last + 1 - at)
        rc = lib.check(at, count, found.data_ptr(), found.data_ptr() + 8, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        at += count
    n, which = found.tolist()
    assert n == 0, f"{n} reciprocals differ, one of them at bits {which:#x}"
