"""The native launch sequences (csrc/sequence.cu) on the CPU: compiled against stubs that record the calls, with the argument
structures laid out as ctypes lays them out."""

import ctypes
import re
import subprocess
from pathlib import Path

import pytest

from dist_moe_b200 import _call, _native

ROOT = Path(__file__).resolve().parents[1]
HEADER = (ROOT / "include" / "dist_moe_b200.h").read_text()


@pytest.fixture(scope="module")
def stub(tmp_path_factory):
    """sequence.cu with every library call it makes replaced by one that appends its name and answers `fail_at`'s code."""
    work = tmp_path_factory.mktemp("sequence")
    source = (ROOT / "dist_moe_b200" / "csrc" / "sequence.cu").read_text()
    called = sorted(set(re.findall(r"\b(dm_\w+)\(", source)) - {"dm_bf16_forward", "dm_bf16_backward", "dm_mxfp8_forward",
                                                                 "dm_mxfp8_backward"})
    # each call is recorded by name and, in a second log, with its barrier's pads and its predicate (pointers as numbers)
    code = ['#include <string>', '#include "../../include/dist_moe_b200.h"', "static std::string calls, details, fail;",
            'extern "C" const char* stub_calls() { return calls.c_str(); }',
            'extern "C" const char* stub_details() { return details.c_str(); }',
            'extern "C" void stub_reset(const char* f) { calls.clear(); details.clear(); fail = f; }',
            "static int note(const char* n, const void* pads, const void* cond) {",
            "  calls += n; calls += ' ';",
            "  details += std::string(n) + ',' + std::to_string((unsigned long)pads) + ',' + std::to_string((unsigned long)cond) + ' ';",
            "  return fail == n ? 7 : 0; }"]
    for name in called:
        text = re.search(r"^int " + name + r"\(.*?\);", HEADER, flags=re.M | re.S).group(0)[:-1]
        words = re.findall(r"\w+", text)
        pads = "signal_pads" if "signal_pads" in words else "nullptr"
        cond = next((w for w in ("cond", "save_cond", "use_alt") if w in words), "nullptr")
        answer = "return 1;" if name == "dm_route_decode_kernel_enabled" else f'return note("{name}", {pads}, {cond});'
        code.append(f'extern "C" {text} {{ {answer} }}')
    src = work / "a" / "csrc"
    src.mkdir(parents=True)
    (work / "include").mkdir()
    (work / "include" / "dist_moe_b200.h").write_text(HEADER)
    (src / "stub.cpp").write_text("\n".join(code))
    (src / "sequence.cpp").write_text(source.replace("#include <cuda_runtime.h>\n", ""))
    out = work / "stub.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-o", str(out), str(src / "stub.cpp"), str(src / "sequence.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(out))
    lib.stub_calls.restype = lib.stub_details.restype = ctypes.c_char_p
    return lib


DISPATCH_PADS, COMBINE_PADS, COND = 0xD0, 0xC0, 0xCD


def _run(lib, name, steps, fail="", ep=1, **fields):
    context, call, report = _native.LayerContext(), _native.LayerCall(), (ctypes.c_int32 * 2)()
    context.ep, context.e_local, context.T_max = ep, 4, 64
    context.dispatch_pads, context.combine_pads = DISPATCH_PADS, COMBINE_PADS
    call.T, call.cond = 64, COND
    for key, value in fields.items():
        setattr(call, key, value)
    lib.stub_reset(fail.encode())
    fn = getattr(lib, name)
    fn.argtypes, fn.restype = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p], ctypes.c_int
    rc = fn(ctypes.addressof(context), ctypes.addressof(call), steps, ctypes.addressof(report), None)
    return rc, lib.stub_calls().decode().split(), list(report)


@pytest.mark.parametrize("struct,cls", [("dm_layer_context", _native.LayerContext), ("dm_layer_call", _native.LayerCall)])
def test_structures_match_the_header(struct, cls, tmp_path):
    names = [f[0] for f in cls._fields_]
    lines = "\n".join(f'printf("%zu ", offsetof({struct}, {n}));' for n in names)
    (tmp_path / "p.cpp").write_text(f'#include <cstddef>\n#include <cstdio>\n#include "{ROOT}/include/dist_moe_b200.h"\n'
                                    f'int main() {{ {lines} printf("%zu", sizeof({struct})); }}')
    subprocess.run(["g++", "-o", str(tmp_path / "p"), str(tmp_path / "p.cpp")], check=True)
    got = [int(v) for v in subprocess.run([str(tmp_path / "p")], capture_output=True, text=True, check=True).stdout.split()]
    assert got == [getattr(cls, n).offset for n in names] + [ctypes.sizeof(cls)]


def test_step_names_match_the_header():
    for prefix, table in (("DM_FWD_", _call.FWD), ("DM_BWD_", _call.BWD)):
        declared = {n.lower(): int(v) for n, v in re.findall(prefix + r"(\w+) = (\d+)", HEADER)}
        assert declared == table


BF16_FWD = ("publish route plan_fwd_bf16 cond_copy gemm_fprop_dispatch swiglu_fwd gemm_fprop scale_and_sum").split()
BF16_BWD = ("plan_bwd_bf16 cond_copy gemm_fprop_dispatch swiglu_fwd gemm_fprop cond_copy broadcast_and_scale gemm_dgrad_dispatch "
            "gemm_wgrad swiglu_bwd gemm_dgrad gemm_wgrad scale_and_sum").split()
MX_FWD = ("publish route_counted plan_fwd_blockscaled cond_copy quant_mxfp8_rowcol_gather_at gemm_blockscaled_counted "
          "swiglu_fwd_quant_mxfp8_rowcol_at gemm_blockscaled_counted scale_and_sum").split()
MX_BWD = ("plan_bwd_blockscaled cond_copy quant_mxfp8_rowcol_gather_at gemm_blockscaled_counted "
          "swiglu_fwd_quant_mxfp8_rowcol_at gemm_blockscaled_counted cond_copy broadcast_and_scale "
          "quant_mxfp8_rowcol_gather_at gemm_blockscaled_dgrad_counted gemm_blockscaled_wgrad_compact "
          "swiglu_bwd_quant_mxfp8_at gemm_blockscaled_dgrad_counted gemm_blockscaled_wgrad_compact scale_and_sum").split()


@pytest.mark.parametrize("name,table,want", [("dm_bf16_forward", _call.FWD, BF16_FWD), ("dm_bf16_backward", _call.BWD, BF16_BWD),
                                             ("dm_mxfp8_forward", _call.FWD, MX_FWD), ("dm_mxfp8_backward", _call.BWD, MX_BWD)])
def test_order_parts_and_failures(stub, name, table, want):
    want = ["dm_" + n for n in want]
    every = sum(table.values())
    rc, calls, report = _run(stub, name, every)
    assert (rc, calls, report) == (0, want, [len(want), 0])
    # the steps one by one, in their order, make the same calls
    parts = [_run(stub, name, bit)[1] for bit in table.values()]
    assert sum(parts, []) == want
    # barriers appear with several ranks only, and count as launches
    rc, calls, report = _run(stub, name, every, ep=2)
    assert [c for c in calls if c != "dm_barrier"] == want and calls.count("dm_barrier") >= 2 and report == [len(calls), 0]
    assert sum([_run(stub, name, bit, ep=2)[1] for bit in table.values()], []) == calls
    # a failing call ends the sequence, and its step is named
    for i, fail in enumerate(want):
        if fail in want[:i]:
            continue
        rc, calls, report = _run(stub, name, every, fail=fail)
        assert rc == 7 and calls == want[:i + 1] and report[0] == i and report[1] in table.values()


# Two ranks: every call with its predicate ("?": only where the planner's decision on this layer says so), and at which pads
# the ranks meet.  Peers read what a barrier stands behind (published rows, expert outputs, their gradients), or have read it
# before the next call overwrites it (the closing one); the two of the recompute block are predicated as it is.
TWO_RANKS = {
    "dm_bf16_forward": "publish barrier:dispatch route plan_fwd_bf16 cond_copy? gemm_fprop_dispatch swiglu_fwd gemm_fprop "
                       "barrier:combine scale_and_sum?",
    "dm_bf16_backward": "plan_bwd_bf16 cond_copy? barrier:dispatch? gemm_fprop_dispatch? swiglu_fwd gemm_fprop? "
                        "barrier:combine? cond_copy? broadcast_and_scale_select? barrier:combine gemm_dgrad_dispatch gemm_wgrad "
                        "swiglu_bwd gemm_dgrad gemm_wgrad barrier:dispatch scale_and_sum",
    "dm_mxfp8_forward": "publish barrier:dispatch route_counted plan_fwd_blockscaled cond_copy? quant_mxfp8_rowcol_gather_at "
                        "gemm_blockscaled_counted swiglu_fwd_quant_mxfp8_rowcol_at gemm_blockscaled_counted barrier:combine "
                        "scale_and_sum?",
    "dm_mxfp8_backward": "plan_bwd_blockscaled cond_copy? barrier:dispatch? quant_mxfp8_rowcol_gather_at? "
                         "gemm_blockscaled_counted? swiglu_fwd_quant_mxfp8_rowcol_at? gemm_blockscaled_counted? "
                         "barrier:combine? cond_copy? broadcast_and_scale_select? barrier:combine quant_mxfp8_rowcol_gather_at "
                         "gemm_blockscaled_dgrad_counted gemm_blockscaled_wgrad_compact swiglu_bwd_quant_mxfp8_at "
                         "gemm_blockscaled_dgrad_counted gemm_blockscaled_wgrad_compact barrier:dispatch scale_and_sum",
}


@pytest.mark.parametrize("name", sorted(TWO_RANKS))
def test_barriers_and_predicates_with_two_ranks(stub, name):
    table = _call.FWD if name.endswith("forward") else _call.BWD
    score = ctypes.c_float()
    options = dict(grad_scores=ctypes.addressof(score), keep_h3=1)

    def shown(steps):
        _run(stub, name, steps, ep=2, **options)
        out = []
        for call, pads, cond in (entry.split(",") for entry in stub.stub_details().decode().split()):
            where = {0: "", DISPATCH_PADS: ":dispatch", COMBINE_PADS: ":combine"}[int(pads)]
            out.append(call.removeprefix("dm_") + where + {0: "", COND: "?"}[int(cond)])
        return out

    assert shown(sum(table.values())) == TWO_RANKS[name].split()
    assert sum([shown(bit) for bit in table.values()], []) == TWO_RANKS[name].split()


def test_options_of_the_bf16_sequences(stub):
    assert "dm_cond_copy" not in _run(stub, "dm_bf16_forward", 255, scratch_only=1)[1]
    assert "dm_swiglu_fwd" not in _run(stub, "dm_bf16_forward", 255, fuse_swiglu=1)[1]
    gathered = _run(stub, "dm_bf16_forward", 255, separate_gather=1)
    assert "dm_gather_rows" in gathered[1] and "dm_gemm_fprop_dispatch" not in gathered[1] and gathered[2][0] == len(gathered[1])
    score = ctypes.c_float()
    select = _run(stub, "dm_bf16_backward", _call.BWD["grad_h3"], grad_scores=ctypes.addressof(score))
    copied = _run(stub, "dm_bf16_backward", _call.BWD["grad_h3"], grad_scores=ctypes.addressof(score), h3_in_combine=1)
    assert select[1] == ["dm_broadcast_and_scale_select"] and copied[1] == ["dm_broadcast_and_scale"]
