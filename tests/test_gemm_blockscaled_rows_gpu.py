"""MXFP8 GEMMs over routed rows (pairs of CTAs, rows on the MMA's N side) at the edges of their tiles: experts of no
row, of one row, of one row more than a step of 32, an atom of 128 and a tile of 256, tiles that start inside a scale atom,
and an odd number of 128-column blocks.  References and bounds as in test_gemm_blockscaled_gpu."""

import pytest
import torch

from tests.test_gemm_blockscaled_gpu import _close, _nat, _quant_act, _tile32_weight
from tests.test_gemm_blockscaled_swapped_gpu import _operands

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
COUNTS = [[1, 0, 33, 128, 129], [256, 257, 31], [300, 545, 0, 64], [1040]]


def _op(nat, t):
    return nat.Operand(t.data_ptr(), t.numel() * t.element_size(), None) if t is not None else nat.Operand(None, 0, None)


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("K,N", [(256, 384), (1280, 256)])
def test_dense_and_scattered_rows(counts, K, N):
    nat, fmt = _nat(), 0
    E, off, real, R, (qa, sa, da, inv), (qw, sw, dw, einv), offs, cnts = _operands(nat, fmt, counts, K, N, 3 * fmt + K)
    status = torch.zeros(8, dtype=torch.int32, device=DEV)
    out = torch.full((R + 8, N), 5.0, device=DEV, dtype=torch.bfloat16)
    sct = torch.full((R, N), 5.0, device=DEV, dtype=torch.bfloat16)
    perm = torch.randperm(R, device=DEV)
    ptrs = torch.zeros(R, dtype=torch.int64, device=DEV)
    ptrs[real.to(DEV)] = sct.data_ptr() + perm[real.to(DEV)].to(torch.int64) * (N * 2)
    for dst, table in ((out, None), (None, ptrs)):
        rc = nat.lib.dm_gemm_blockscaled_counted(fmt, _op(nat, qa), _op(nat, sa), qw.data_ptr(), sw.data_ptr(), _op(nat, dst),
                                                 _op(nat, None), nat.ptr(table), _op(nat, inv), nat.ptr(einv),
                                                 offs.data_ptr(), cnts.data_ptr(), E, R, N, K, 0, 0, 1.0, 0.0, None, 0,
                                                 status.data_ptr(), nat.stream_ptr())
        nat.check(rc, "dm_gemm_blockscaled_counted")
    torch.cuda.synchronize()
    assert status[0].item() == 0, status.tolist()
    got, touched = sct.cpu(), torch.zeros(R, dtype=torch.bool)
    for e, n in enumerate(counts):
        rows = torch.arange(off[e], off[e] + n)
        if n:
            _close(out.cpu()[rows], da[rows] @ dw[e].T, f"expert {e}")
            touched[perm.cpu()[rows]] = True
            assert torch.equal(got[perm.cpu()[rows]], out.cpu()[rows])
        assert bool((out[off[e] + n:off[e + 1]] == 0).all()), "padding rows of a dense result are zero"
    assert bool((out[off[-1]:] == 5.0).all()) and bool((got[~touched] == 5.0).all())


@pytest.mark.parametrize("counts", COUNTS)
def test_swiglu_rows(counts):
    """h1, h2 and the quantised h2, at 2F = 384: the last pair of column blocks is half empty."""
    nat, fmt = _nat(), 0
    K, F = 512, 192
    N = 2 * F
    E, off, real, R, (qa, sa, da, inv), (qw, sw, dw, einv), offs, cnts = _operands(nat, fmt, counts, K, N, 17 + fmt, F)
    status = torch.zeros(8, dtype=torch.int32, device=DEV)
    h1 = torch.full((R, N), 5.0, device=DEV, dtype=torch.bfloat16)
    h2 = torch.full((R, F), 5.0, device=DEV, dtype=torch.bfloat16)
    st = nat.stream_ptr()
    nat.check(nat.lib.dm_gemm_blockscaled_counted(fmt, _op(nat, qa), _op(nat, sa), qw.data_ptr(), sw.data_ptr(), _op(nat, h1),
                                                  _op(nat, h2), None, _op(nat, inv), nat.ptr(einv), offs.data_ptr(),
                                                  cnts.data_ptr(), E, R, N, K, 1, 0, 1.702, 7.0, None, 0,
                                                  status.data_ptr(), st), "swiglu")
    atoms = (F // 32 + 3) // 4
    want_q, want_s = torch.zeros(R, F, dtype=torch.uint8, device=DEV), torch.zeros(R * atoms * 4, dtype=torch.uint8, device=DEV)
    got_q, got_s = torch.zeros_like(want_q), torch.zeros_like(want_s)
    live = torch.zeros(R, dtype=torch.int64, device=DEV)
    live[real.to(DEV)] = 1
    rows = torch.tensor([R], dtype=torch.int32, device=DEV)
    nat.check(nat.lib.dm_quant_mxfp8_row_live(live.data_ptr(), h2.data_ptr(), rows.data_ptr(), R, F, want_q.data_ptr(), 0,
                                              want_s.data_ptr(), 0, 1, st), "row")
    nat.check(nat.lib.dm_gemm_blockscaled_swiglu_mxfp8_counted(_op(nat, qa), _op(nat, sa), qw.data_ptr(), sw.data_ptr(),
                                                               _op(nat, got_q), _op(nat, got_s), offs.data_ptr(),
                                                               cnts.data_ptr(), E, R, N, K, 0, 1.702, 7.0, None, 0,
                                                               status.data_ptr(), st), "swiglu + quant")
    torch.cuda.synchronize()
    assert status[0].item() == 0, status.tolist()
    idx = torch.stack([torch.arange(F).reshape(-1, 8), torch.arange(F).reshape(-1, 8) + F], dim=1).reshape(-1)
    inv_idx = torch.empty_like(idx)
    inv_idx[idx] = torch.arange(N)
    pad = torch.ones(R, dtype=torch.bool)
    pad[real] = False
    h1c, h2c = h1.cpu(), h2.cpu()
    for e, n in enumerate(counts):
        rows = torch.arange(off[e], off[e] + n)
        if n:
            _close(h1c[rows], (da[rows] @ dw[e].T)[:, inv_idx], f"h1 expert {e}")
            g, u = h1c[rows, :F].float(), h1c[rows, F:].float()
            _close(h2c[rows], g * torch.sigmoid(g) * u, f"h2 expert {e}")
    assert bool((h1c[pad] == 5.0).all()) and bool((h2c[pad] == 5.0).all())
    assert torch.equal(got_q, want_q) and torch.equal(got_s, want_s)


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("K,N", [(256, 384), (640, 256)])
def test_input_gradient_rows(counts, K, N):
    nat = _nat()
    off = [0]
    for n in counts:
        off.append(off[-1] + (n + 127) // 128 * 128)
    E, R = len(counts), max(off[-1], 128)
    torch.manual_seed(K + N)
    dy = torch.zeros(R, K, device=DEV, dtype=torch.bfloat16)
    for e, n in enumerate(counts):
        dy[off[e]:off[e] + n] = torch.randn(n, K, device=DEV).bfloat16()
    w = (torch.randn(E, K, N, device=DEV) * 0.05).bfloat16()
    qa, sa, da, _ = _quant_act(nat, dy, 0)
    qw, _, s_dgrad, dw = _tile32_weight(nat, w)
    offs = torch.tensor(off, dtype=torch.int32, device=DEV)
    cnts = torch.tensor(counts, dtype=torch.int32, device=DEV)
    status = torch.zeros(8, dtype=torch.int32, device=DEV)
    out = torch.full((R + 8, N), 5.0, device=DEV, dtype=torch.bfloat16)
    nat.check(nat.lib.dm_gemm_blockscaled_dgrad_counted(_op(nat, qa), _op(nat, sa), qw.data_ptr(), s_dgrad.data_ptr(),
                                                        _op(nat, out), None, offs.data_ptr(), cnts.data_ptr(), E, R, N, K,
                                                        None, 0, status.data_ptr(), nat.stream_ptr()), "dgrad")
    torch.cuda.synchronize()
    assert status[0].item() == 0, status.tolist()
    for e, n in enumerate(counts):
        rows = torch.arange(off[e], off[e] + n)
        if n:
            _close(out.cpu()[rows], da[rows] @ dw[e], f"expert {e}")
        assert bool((out[off[e] + n:off[e + 1]] == 0).all())
    assert bool((out[off[-1]:] == 5.0).all())


@pytest.mark.parametrize("swapped,fmt", [(False, 0), (True, 0), (True, 1)])
@pytest.mark.parametrize("counted", [True, False])
def test_groups_that_are_not_padded_are_left_out(swapped, fmt, counted):
    """Experts that do not start on 128 rows: a status, none of their rows written, the others as ever."""
    nat = _nat()
    K, N = 512, 256
    E, off, real, R, (qa, sa, da, inv), (qw, sw, dw, einv), _, _ = _operands(nat, fmt, [128, 128, 128, 128], K, N, 23 + fmt)
    off = [0, 128, 160, 384, 512]
    offs = torch.tensor(off, dtype=torch.int32, device=DEV)
    cnts = torch.tensor([100, 32, 200, 128], dtype=torch.int32, device=DEV)
    status = torch.zeros(8, dtype=torch.int32, device=DEV)
    out = torch.full((R, N), 5.0, device=DEV, dtype=torch.bfloat16)
    fn = nat.lib.dm_gemm_blockscaled_swapped if swapped else nat.lib.dm_gemm_blockscaled_counted
    nat.check(fn(fmt, _op(nat, qa), _op(nat, sa), qw.data_ptr(), sw.data_ptr(), _op(nat, out), _op(nat, None), None,
                 _op(nat, inv), nat.ptr(einv), offs.data_ptr(), cnts.data_ptr() if counted else None, E, R, N, K, 0, 0, 1.0,
                 0.0, None, 0, status.data_ptr(), nat.stream_ptr()), "unpadded group")
    torch.cuda.synchronize()
    assert status.tolist()[:4] == [2, -1, 2, 160]
    got = out.cpu()
    assert bool((got[160:384] == 5.0).all())
    for e, rows in ((0, 100), (1, 32), (3, 128)):
        at = torch.arange(off[e], off[e] + rows)
        _close(got[at], da[at] @ dw[e].T, f"expert {e}")


@pytest.mark.parametrize("offset", [16, 112, 128, 656])
@pytest.mark.parametrize("form", ["forward", "swiglu", "input gradient"])
def test_scales_at_any_sixteen_bytes(form, offset):
    """The rows' scales may start at any multiple of 16 bytes, and their extent need not be told: the entry points' older
    kernel copied them by address.  Same bits as from the start of an allocation."""
    nat = _nat()
    counts, K, N = [300, 0, 33, 128], 1280, 256
    E, off, real, R, (qa, sa, _, _), (qw, sw, _, _), offs, cnts = _operands(nat, 0, counts, K, N, 41)
    if form == "input gradient":
        w = (torch.randn(E, K, N, device=DEV) * 0.05).bfloat16()
        qw, _, sw, _ = _tile32_weight(nat, w)
    n = sa.numel()
    wide = torch.full((n + 1024,), 0x55, dtype=torch.uint8, device=DEV)
    wide[offset:offset + n] = sa.view(torch.uint8).reshape(-1)
    at = torch.tensor([offset], dtype=torch.int64, device=DEV)
    results = []
    for scales in (_op(nat, sa), nat.Operand(wide.data_ptr(), wide.numel(), at.data_ptr()), nat.Operand(wide.data_ptr(), 0, at.data_ptr())):
        status = torch.zeros(8, dtype=torch.int32, device=DEV)
        out = torch.full((R, N // 2 if form == "swiglu" else N), 5.0, device=DEV, dtype=torch.bfloat16)
        none, tail = _op(nat, None), (None, 0, status.data_ptr(), nat.stream_ptr())
        if form == "input gradient":
            rc = nat.lib.dm_gemm_blockscaled_dgrad(_op(nat, qa), scales, qw.data_ptr(), sw.data_ptr(), _op(nat, out), None,
                                                   offs.data_ptr(), E, R, N, K, *tail)
        else:
            swiglu = form == "swiglu"
            rc = nat.lib.dm_gemm_blockscaled(0, _op(nat, qa), scales, qw.data_ptr(), sw.data_ptr(), none if swiglu else _op(nat, out),
                                             _op(nat, out) if swiglu else none, None, none, None, offs.data_ptr(), E, R, N, K,
                                             int(swiglu), 0, 1.0, 0.0, *tail)
        nat.check(rc, form)
        torch.cuda.synchronize()
        assert status[0].item() == 0, status.tolist()
        results.append(out)
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])
    assert bool((results[0][real.to(DEV)] != 5.0).any())


class _Launch:
    """One launch of the pair kernel in any of its forms, its operands at device offsets inside wider buffers."""

    FORMS = ("dense", "scattered", "swiglu", "swiglu quantised", "input gradient")

    def __init__(self, form, counts, K, N, offset):
        nat, self.form = _nat(), form
        self.nat, self.K, self.N, self.F = nat, K, N, N // 2
        self.E, self.off, self.real, self.R, (qa, sa, _, _), (qw, sw, _, _), self.offs, self.cnts = _operands(
            nat, 0, counts, K, N, 57 + N, N // 2 if form.startswith("swiglu") else None)
        if form == "input gradient":
            qw, _, sw, _ = _tile32_weight(nat, (torch.randn(self.E, K, N, device=DEV) * 0.05).bfloat16())
        self.qw, self.sw, self.offset = qw, sw, offset
        self.at = torch.tensor([offset], dtype=torch.int64, device=DEV)
        self.qa, self.sa = self._placed(qa.view(torch.uint8).reshape(-1)), self._placed(sa.view(torch.uint8).reshape(-1))
        atoms = (self.F // 32 + 3) // 4
        self.sizes = {"dense": [self.R * N * 2], "input gradient": [self.R * N * 2], "scattered": [self.R * N * 2],
                      "swiglu": [self.R * N * 2, self.R * self.F * 2],
                      "swiglu quantised": [self.R * self.F, self.R * atoms * 4]}[form]

    def _placed(self, data):
        wide = torch.full((data.numel() + 2 * self.offset + 1024,), 0x7F, dtype=torch.uint8, device=DEV)
        wide[self.offset:self.offset + data.numel()] = data
        return wide

    def _at(self, t):
        return self.nat.Operand(t.data_ptr(), t.numel(), self.at.data_ptr())

    def run(self, num_sms, cond=None):
        """The result bytes, poisoned before the launch, with those around them."""
        nat, none = self.nat, self.nat.Operand(None, 0, None)
        out = [torch.full((n + 2 * self.offset + 1024,), 0x7F, dtype=torch.uint8, device=DEV) for n in self.sizes]
        status = torch.zeros(8, dtype=torch.int32, device=DEV)
        tail = (nat.ptr(cond), num_sms, status.data_ptr(), nat.stream_ptr())
        head = (self._at(self.qa), self._at(self.sa), self.qw.data_ptr(), self.sw.data_ptr())
        shape = (self.offs.data_ptr(), self.cnts.data_ptr(), self.E, self.R, self.N, self.K)
        if self.form == "input gradient":
            rc = nat.lib.dm_gemm_blockscaled_dgrad_counted(*head, self._at(out[0]), None, *shape, *tail)
        elif self.form == "swiglu quantised":
            rc = nat.lib.dm_gemm_blockscaled_swiglu_mxfp8_counted(*head, self._at(out[0]), self._at(out[1]), *shape, 0, 1.0, 0.0,
                                                                  *tail)
        else:
            swiglu, ptrs = self.form == "swiglu", None
            if self.form == "scattered":
                ptrs = torch.zeros(self.R, dtype=torch.int64, device=DEV)
                rows = self.real.to(DEV)
                ptrs[rows] = out[0].data_ptr() + self.offset + rows.flip(0) * (self.N * 2)
            rc = nat.lib.dm_gemm_blockscaled_counted(0, *head, none if ptrs is not None else self._at(out[0]),
                                                     self._at(out[1]) if swiglu else none, nat.ptr(ptrs), none, None, *shape,
                                                     int(swiglu), 0, 1.0, 0.0, *tail)
        nat.check(rc, self.form)
        torch.cuda.synchronize()
        assert status[0].item() == 0, status.tolist()
        return out


@pytest.mark.parametrize("form", _Launch.FORMS)
@pytest.mark.parametrize("counts", [[256, 512, 100, 0, 257], [96, 33, 128, 64, 1, 120], [300, 545, 0, 64, 180]],
                         ids=["shared columns", "one atom", "inside atoms"])
@pytest.mark.parametrize("K", [256, 1152])
def test_several_tiles_per_pair(form, counts, K):
    """Pairs that take many tiles in turn: both accumulators, their shared columns, the ring running on from tile to tile.  The
    bits of the launch that gives every tile a pair of its own, and nothing written beside the results."""
    one_each = _Launch(form, counts, K, 768, 0).run(0)
    several = _Launch(form, counts, K, 768, 0)
    for num_sms in (1, 2, 5, 2):
        for a, b in zip(one_each, several.run(num_sms)):
            assert torch.equal(a, b), num_sms


@pytest.mark.parametrize("form", _Launch.FORMS)
def test_device_offsets_and_a_false_predicate(form):
    """Operands and results that start inside an allocation, at an offset read on the device: the same bits there, none around
    them.  Where the predicate is false nothing is written."""
    plain, moved = (_Launch(form, [200, 0, 300, 31], 512, 384, offset) for offset in (0, 128 * 37))
    yes, no = (torch.tensor([v], dtype=torch.int32, device=DEV) for v in (1, 0))
    for size, a, b, c in zip(plain.sizes, plain.run(0), moved.run(0), moved.run(4, cond=yes)):
        assert torch.equal(b[moved.offset:moved.offset + size], a[:size]) and torch.equal(b, c)
        assert bool((b[:moved.offset] == 0x7F).all()) and bool((b[moved.offset + size:] == 0x7F).all())
    for t in moved.run(0, cond=no):
        assert bool((t == 0x7F).all())
