"""Rules that every kernel source keeps, checked on the text (CPU)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "dist_moe_b200" / "csrc"


def _kernels():
    """(name, body) of every __global__ function."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            begin = text.index("{", text.index(")", text.index("_kernel", m.end())))
            depth, i = 0, begin
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            yield re.search(r"(\w+_kernel)\b", text[m.end():]).group(1), text[begin:i]


KERNELS = dict(_kernels())


@pytest.mark.parametrize("name", sorted(n for n, body in KERNELS.items() if "bulk_commit()" in body))
def test_bulk_stores_are_waited_for_before_the_block_ends(name):
    """A block that ends gives its shared memory back; a bulk store that has not read its staged box yet would store another
    block's bytes."""
    body = KERNELS[name]
    assert "bulk_wait_all()" in body[body.rindex("bulk_commit()"):]


def test_the_kernels_were_found():
    assert {"wgrad_gemm_kernel", "blockscaled_wide_kernel", "rows_gemm_kernel", "blockscaled_swapped_kernel"} <= set(KERNELS)
