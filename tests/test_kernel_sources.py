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


@pytest.mark.parametrize("name", sorted(n for n, body in KERNELS.items() if "mbar_wait(" in body))
def test_a_wait_that_runs_out_is_recorded(name):
    """A kernel that may give up waiting says so."""
    assert "set_status(" in KERNELS[name]


def test_rows_fetched_by_hand_are_those_the_thread_reads():
    """Where a bulk copy of a token's rows does not come in time, nothing lies between a thread's own fetch and its reads: the pieces
    that it fetches, walked over as the kernel does, have to be the ones that it reads."""
    body = KERNELS["rmsnorm_combine_fwd_staged_kernel"]
    fetch = re.search(r"if \(!mbar_wait\([^\n]*\n(.*?)src\[(.*?)\] = ", body, re.S)
    loops, index = re.findall(r"for \(int (\w+) = ([\w.]+); \w+ < (\w+); (?:\+\+\w+|\w+ \+= (\d+))\)", fetch[1]), fetch[2]
    assert loops and index

    def walk(todo, names):
        if not todo:
            return {eval(index, {}, names)}
        (name, first, end, step), rest = todo[0], todo[1:]
        first = names["thread"] if first == "threadIdx.x" else int(first)
        return set().union(*(walk(rest, {**names, name: i}) for i in range(first, names[end], int(step or 1))))

    for K, vec in [(1, 32), (4, 352), (3, 256), (8, 896), (5, 1)]:
        for thread in (0, 1, 31, 255):
            reads = {k * vec + v for k in range(K) for v in range(thread, vec, 256)}
            assert walk(loops, {"K": K, "vec": vec, "rows": K * vec, "thread": thread}) == reads, (K, vec, thread)


def test_two_buffers_only_where_two_blocks_of_them_fit():
    """The rule of dm_rmsnorm_combine_fwd, evaluated from its own expressions for every K x D: a block per SM with two buffers leaves
    the SM to a single block where three with one buffer would fit."""
    text = (CSRC / "rmsnorm.cu").read_text()
    text = text[text.index("auto choose ="):]

    def python(source):
        return re.sub(r"(.*) \? (\S+) : (\S+)", r"(\2 if \1 else \3)", source.replace("kNormStaged", "216 * 1024").replace(" / ", " // "))

    buffers_rule = python(re.search(r"const int buffers = (.*?);", text)[1])
    fit_rule = python(re.search(r"const int64_t fit = (.*?);", text)[1])
    helper = re.search(r"auto resident = .*? return (.*?); \};", text)
    for elements in range(8, 216 * 1024 // 2 + 1, 8):
        names = {"bytes": 2 * elements}
        if helper:
            names["resident"] = lambda buffers: eval(python(helper[1]), {}, {"bytes": 2 * elements, "buffers": buffers})
        names["buffers"] = eval(buffers_rule, {}, names)
        fit = eval(fit_rule, {}, names)
        assert fit >= names["buffers"], (elements, names["buffers"], fit)
        assert fit * (names["buffers"] * 2 * elements + 4096) <= 227 * 1024 - 1024 + 4096 * (fit == 1)
