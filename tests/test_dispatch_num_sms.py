"""``num_sms`` of the launches: the mark that the counters of a fused dispatch are kept clear goes to the dispatch GEMMs of a context and
to no other launch, and no bound on the SMs that a caller may have given before is taken for it."""

import ctypes
import re
import subprocess
from pathlib import Path

import pytest
import torch

from dist_moe_b200 import _call, _native

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "dist_moe_b200" / "csrc"
HEADER = (ROOT / "include" / "dist_moe_b200.h").read_text()
MARK = _native.GATHER_FLAGS_KEPT_CLEAR


@pytest.fixture(scope="module")
def sequence(tmp_path_factory):
    """sequence.cu with every library call that it makes replaced by one that notes its name and its num_sms."""
    work = tmp_path_factory.mktemp("num_sms")
    source = (CSRC / "sequence.cu").read_text()
    own = {"dm_bf16_forward", "dm_bf16_backward", "dm_mxfp8_forward", "dm_mxfp8_backward"}
    code = ['#include <string>', '#include "../../include/dist_moe_b200.h"', "static std::string notes;",
            'extern "C" const char* stub_notes() { return notes.c_str(); }', 'extern "C" void stub_reset() { notes.clear(); }',
            'static int note(const char* n, long v) { notes += std::string(n) + "," + std::to_string(v) + " "; return 0; }']
    for name in sorted(set(re.findall(r"\b(dm_\w+)\(", source)) - own):
        text = re.search(r"^int " + name + r"\(.*?\);", HEADER, flags=re.M | re.S).group(0)[:-1]
        body = f'return note("{name}", num_sms);' if re.search(r"\bnum_sms\b", text) else "return 0;"
        code.append(f'extern "C" {text} {{ {body} }}')
    src = work / "a" / "csrc"
    src.mkdir(parents=True)
    (work / "include").mkdir()
    (work / "include" / "dist_moe_b200.h").write_text(HEADER)
    (src / "stub.cpp").write_text("\n".join(code))
    (src / "sequence.cpp").write_text(source.replace("#include <cuda_runtime.h>\n", ""))
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-o", str(work / "s.so"), str(src / "stub.cpp"), str(src / "sequence.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(work / "s.so"))
    lib.stub_notes.restype = ctypes.c_char_p

    def run(name, steps, num_sms, kept):
        context, call, report = _native.LayerContext(), _native.LayerCall(), (ctypes.c_int32 * 2)()
        context.ep, context.e_local, context.T_max, context.num_sms, context.gather_flags_kept_clear = 1, 4, 64, num_sms, kept
        call.T = 64
        lib.stub_reset()
        fn = getattr(lib, name)
        fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p]
        assert fn(ctypes.addressof(context), ctypes.addressof(call), steps, ctypes.addressof(report), None) == 0
        return [(n, int(v)) for n, v in (item.split(",") for item in lib.stub_notes().decode().split())]

    return run


@pytest.mark.parametrize("num_sms", [0, 1, 148, 70_000, 2**31 - 1, -1])
@pytest.mark.parametrize("kept", [0, 1])
def test_only_dispatch_launches_carry_the_mark(sequence, num_sms, kept):
    want = MARK | min(max(num_sms, 0), 0xffff)
    dispatches = 0
    for name, steps in [("dm_bf16_forward", _call.FWD), ("dm_bf16_backward", _call.BWD), ("dm_mxfp8_forward", _call.FWD),
                        ("dm_mxfp8_backward", _call.BWD)]:
        noted = sequence(name, sum(steps.values()), num_sms, kept)
        assert noted
        for launch, value in noted:
            marked = kept and launch.endswith("_dispatch")
            assert value == (want if marked else num_sms), (launch, value)
            dispatches += launch.endswith("_dispatch")
    assert dispatches == 3


def test_what_counts_as_the_mark(tmp_path):
    (tmp_path / "p.cpp").write_text('#include "row_tiles.cuh"\nextern "C" int kept(int n) { return dm::rw_flags_kept_clear(n); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(tmp_path / "p.so"), str(tmp_path / "p.cpp")], check=True)
    kept = ctypes.CDLL(str(tmp_path / "p.so")).kept
    assert all(kept(MARK | n) for n in (0, 1, 148, 0xffff))
    assert not any(kept(n) for n in (0, 1, 148, 0xffff, 1 << 29, MARK + 0x10000, MARK | 1 << 29, 2**31 - 1, -1, -2**31))


@pytest.mark.gpu
@pytest.mark.parametrize("num_sms", [2**31 - 1, 148, 0])
def test_a_large_bound_leaves_the_clearing_to_the_call(num_sms):
    """The largest bound, on counters that are not clear and one word short of those that are kept clear."""
    dev, rows, n, kd = torch.device("cuda", 0), 300, 256, 128
    torch.manual_seed(0)
    src, w = torch.randn(rows, kd, device=dev).bfloat16(), (torch.randn(2, n, kd, device=dev) * 0.1).bfloat16()
    words = rows // 128 + 2
    flags = torch.full((words + 1,), 77, dtype=torch.int32, device=dev)
    offs = torch.tensor([0, 100, rows], dtype=torch.int32, device=dev)
    ptrs = src.data_ptr() + torch.arange(rows, device=dev) * kd * 2
    a = torch.zeros(rows + 300, kd, device=dev, dtype=torch.bfloat16)
    c, status = torch.zeros(rows, n, device=dev, dtype=torch.bfloat16), torch.zeros(8, dtype=torch.int32, device=dev)
    op = lambda t: _native.Operand(t.data_ptr(), t.numel() * 2, None)  # noqa: E731
    _native.check(_native.lib.dm_gemm_fprop_dispatch(
        ptrs.data_ptr(), flags.data_ptr(), op(a), w.data_ptr(), op(c), _native.Operand(None, 0, None), offs.data_ptr(), 2, rows, n, kd, 0,
        0, 1.0, 0.0, None, num_sms, status.data_ptr(), _native.stream_ptr()), "dispatch")
    torch.cuda.synchronize()
    assert status[0].item() == 0 and flags[words].item() == 77
    assert torch.equal(a[:rows], src)
    want = torch.cat([src[:100].double() @ w[0].double().T, src[100:].double() @ w[1].double().T])
    # fp32 sums of 128 products of bf16 values, rounded to bf16 once
    assert bool(((c.double() - want).abs() <= want.abs() * 2 ** -8 + 1e-4).all())
