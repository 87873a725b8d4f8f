"""CUDA quantisers through the C ABI, bit-exact against the CPU oracle (`oracle/quant.py`), which
is itself held to the reference's Triton quantiser for MXFP8.  Sizes up to the full C3 row width."""

import numpy as np
import pytest
import torch

from oracle import quant as Q

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _nat():
    from dist_moe_b200 import _native

    return _native


def _data(rows, cols, seed, spread=True, specials=True):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, cols, generator=g)
    if spread:
        x = x * torch.logspace(-4, 3, rows)[:, None]
    x = x.bfloat16()
    if specials and rows > 4:
        x[0, :32] = 0
        x[1, 7] = float("inf")
        x[2, 40] = float("nan")
        x[3, :32] = 448.0
    return x


@pytest.mark.parametrize("rows,cols,blocked", [(37, 256, 0), (200, 384, 1), (1000, 4096, 1), (1, 32, 0)])
def test_mxfp8_row(rows, cols, blocked):
    nat = _nat()
    x = _data(rows, cols, rows)
    xd = x.to(DEV)
    q = torch.zeros(rows, cols, dtype=torch.uint8, device=DEV)
    sc = cols // 32
    atoms = (sc + 3) // 4
    n_s = ((rows + 127) // 128 * 128) * atoms * 4 if blocked else rows * sc
    s = torch.full((n_s,), 0xEE, dtype=torch.uint8, device=DEV)
    cnt = torch.tensor([rows], dtype=torch.int32, device=DEV)
    nat.check(nat.lib.dm_quant_mxfp8_row(xd.data_ptr(), cnt.data_ptr(), rows, cols, q.data_ptr(), 0, s.data_ptr(), 0, blocked,
                                         nat.stream_ptr()), "mxfp8_row")
    torch.cuda.synchronize()
    rq, rs = Q.mxfp8_row(x)
    got_s = s.cpu().numpy()
    if blocked:
        r, c = np.meshgrid(np.arange(rows), np.arange(sc), indexing="ij")
        got_s = got_s[Q.blocked_scale_offset(r, c, atoms)]
    else:
        got_s = got_s.reshape(rows, sc)
    np.testing.assert_array_equal(got_s, rs)
    finite = np.repeat(rs != 255, 32, axis=1)
    gq = q.cpu().numpy()
    np.testing.assert_array_equal(gq[finite], rq[finite])
    assert ((gq[~finite] & 0x7F) == 0x7F).all()


@pytest.mark.parametrize("rows,cols", [(96, 64), (333, 520), (4096, 1536)])
def test_mxfp8_col(rows, cols):
    nat = _nat()
    x = _data(rows, cols, rows + 1, specials=False)
    q = torch.zeros(rows, cols, dtype=torch.uint8, device=DEV)
    rb = (rows + 31) // 32
    s = torch.zeros(cols * rb, dtype=torch.uint8, device=DEV)
    nat.check(nat.lib.dm_quant_mxfp8_col(x.to(DEV).data_ptr(), None, rows, cols, q.data_ptr(), s.data_ptr(), 0,
                                         nat.stream_ptr()), "mxfp8_col")
    torch.cuda.synchronize()
    rq, rs = Q.mxfp8_col(x)
    np.testing.assert_array_equal(s.cpu().numpy().reshape(cols, rb), rs)
    np.testing.assert_array_equal(q.cpu().numpy(), rq)


@pytest.mark.parametrize("experts,n,k,blocked", [(2, 64, 96, 0), (3, 256, 512, 1)])
def test_mxfp8_tile32_weights(experts, n, k, blocked):
    nat = _nat()
    w = _data(experts * n, k, 11, spread=False, specials=False) * 0.02
    w = w.bfloat16()
    q = torch.zeros(experts * n, k, dtype=torch.uint8, device=DEV)
    a0, a1 = (k // 32 + 3) // 4, (n // 32 + 3) // 4
    g0 = (n + 127) // 128 * 128 * a0 * 4 if blocked else n * (k // 32)
    g1 = (k + 127) // 128 * 128 * a1 * 4 if blocked else k * (n // 32)
    s0 = torch.zeros(experts * g0, dtype=torch.uint8, device=DEV)
    s1 = torch.zeros(experts * g1, dtype=torch.uint8, device=DEV)
    nat.check(nat.lib.dm_quant_mxfp8_tile32(w.to(DEV).data_ptr(), experts, n, k, q.data_ptr(), s0.data_ptr(),
                                            s1.data_ptr(), blocked, nat.stream_ptr()), "tile32")
    torch.cuda.synchronize()
    gq, g0s, g1s = q.cpu().numpy(), s0.cpu().numpy().reshape(experts, -1), s1.cpu().numpy().reshape(experts, -1)
    for e in range(experts):
        rq, rs = Q.mxfp8_tile32(w[e * n:(e + 1) * n])
        np.testing.assert_array_equal(gq[e * n:(e + 1) * n], rq)
        row_s = np.repeat(rs, 32, axis=0)            # [n, k/32]
        col_s = np.repeat(rs.T, 32, axis=0)          # [k, n/32]
        if blocked:
            r, c = np.meshgrid(np.arange(n), np.arange(k // 32), indexing="ij")
            np.testing.assert_array_equal(g0s[e][Q.blocked_scale_offset(r, c, a0)], row_s)
            r, c = np.meshgrid(np.arange(k), np.arange(n // 32), indexing="ij")
            np.testing.assert_array_equal(g1s[e][Q.blocked_scale_offset(r, c, a1)], col_s)
        else:
            np.testing.assert_array_equal(g0s[e].reshape(n, k // 32), row_s)
            np.testing.assert_array_equal(g1s[e].reshape(k, n // 32), col_s)


@pytest.mark.parametrize("rows,cols", [(33, 256), (128, 7168), (5, 2880 - 2880 % 16)])
def test_nvfp4_token_dense_and_packed_rows(rows, cols):
    nat = _nat()
    x = _data(rows, cols, rows + 2, specials=False)
    xd = x.to(DEV)
    rp, rs, rinv = Q.nvfp4_token_rows(x)
    # dense outputs
    q = torch.zeros(rows, cols // 2, dtype=torch.uint8, device=DEV)
    s = torch.zeros(rows, cols // 16, dtype=torch.uint8, device=DEV)
    inv = torch.zeros(rows, dtype=torch.float32, device=DEV)
    nat.check(nat.lib.dm_quant_nvfp4_token(xd.data_ptr(), None, rows, cols, q.data_ptr(), cols // 2, s.data_ptr(),
                                           cols // 16, 0, inv.data_ptr(), 4, nat.stream_ptr()), "nvfp4_token")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(inv.cpu().numpy().view(np.uint32), rinv.view(np.uint32))
    np.testing.assert_array_equal(s.cpu().numpy(), rs)
    np.testing.assert_array_equal(q.cpu().numpy(), rp)
    # packed dispatch row [q | scales | inv | pad16]: bit-identical to the dense call
    stride = (cols // 2 + cols // 16 + 4 + 15) // 16 * 16
    packed = torch.zeros(rows, stride, dtype=torch.uint8, device=DEV)
    base = packed.data_ptr()
    nat.check(nat.lib.dm_quant_nvfp4_token(xd.data_ptr(), None, rows, cols, base, stride, base + cols // 2, stride, 0,
                                           base + cols // 2 + cols // 16, stride, nat.stream_ptr()), "nvfp4_token")
    torch.cuda.synchronize()
    p = packed.cpu().numpy()
    np.testing.assert_array_equal(p[:, : cols // 2], rp)
    np.testing.assert_array_equal(p[:, cols // 2 : cols // 2 + cols // 16], rs)
    got_inv = np.ascontiguousarray(p[:, cols // 2 + cols // 16 : cols // 2 + cols // 16 + 4]).view(np.uint32)[:, 0]
    np.testing.assert_array_equal(got_inv, rinv.view(np.uint32))


def test_nvfp4_weight_and_swizzle():
    nat = _nat()
    experts, n, k = 3, 160, 256
    g = torch.Generator().manual_seed(7)
    w = (torch.randn(experts, n, k, generator=g) * 0.02).bfloat16()
    rp, rs, gs, gsi = Q.nvfp4_weight(w)
    wd = w.to(DEV)
    amax = torch.linalg.vector_norm(wd, ord=float("inf"), dim=(-2, -1), dtype=torch.float32).clamp(min=1e-12)
    gsd = 2688.0 * torch.reciprocal(amax)
    np.testing.assert_array_equal(gsd.cpu().numpy().view(np.uint32), gs.view(np.uint32))
    q = torch.zeros(experts, n, k // 2, dtype=torch.uint8, device=DEV)
    s = torch.zeros(experts * n, k // 16, dtype=torch.uint8, device=DEV)
    nat.check(nat.lib.dm_quant_nvfp4_weight(wd.data_ptr(), gsd.data_ptr(), experts, n, k, q.data_ptr(), s.data_ptr(), 0,
                                            nat.stream_ptr()), "nvfp4_weight")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(s.cpu().numpy().reshape(experts, n, k // 16), rs)
    np.testing.assert_array_equal(q.cpu().numpy(), rp)
    # swizzle natural -> blocked equals the oracle's layout, padding zeroed
    sw = torch.full(((n + 127) // 128 * 128 * 4 * 4,), 0xEE, dtype=torch.uint8, device=DEV)
    nat.check(nat.lib.dm_sf_swizzle(s[:n].contiguous().data_ptr(), sw.data_ptr(), n, k // 16, nat.stream_ptr()), "swz")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(sw.cpu().numpy(), Q.to_blocked(rs[0]))


@pytest.mark.parametrize("rows,cols,cap", [(96, 64, 128), (333, 512, 384), (4096, 1536, 4096)])
def test_mxfp8_rowcol_equals_the_separate_kernels(rows, cols, cap):
    """One pass producing both copies is bit-identical to the row kernel (blocked scales) and the column kernel
    (blocked scales), which are held to the oracle above."""
    nat = _nat()
    x = _data(rows, cols, rows + 3, specials=False).to(DEV)
    cnt = torch.tensor([rows], dtype=torch.int32, device=DEV)
    ra, ca = (cols // 32 + 3) // 4, ((cap + 31) // 32 + 3) // 4
    n_rs, n_cs = (cap + 127) // 128 * 128 * ra * 4, (cols + 127) // 128 * 128 * ca * 4
    st = nat.stream_ptr()
    q_r = torch.zeros(cap, cols, dtype=torch.uint8, device=DEV)
    s_r = torch.zeros(n_rs, dtype=torch.uint8, device=DEV)
    q_c = torch.zeros(cap, cols, dtype=torch.uint8, device=DEV)
    s_c = torch.zeros(n_cs, dtype=torch.uint8, device=DEV)
    nat.check(nat.lib.dm_quant_mxfp8_row(x.data_ptr(), cnt.data_ptr(), cap, cols, q_r.data_ptr(), 0, s_r.data_ptr(), 0, 1, st), "row")
    nat.check(nat.lib.dm_quant_mxfp8_col(x.data_ptr(), cnt.data_ptr(), cap, cols, q_c.data_ptr(), s_c.data_ptr(), 1, st), "col")
    f_r, fs_r, f_c, fs_c = (torch.zeros_like(t) for t in (q_r, s_r, q_c, s_c))
    nat.check(nat.lib.dm_quant_mxfp8_rowcol(x.data_ptr(), cnt.data_ptr(), cap, cols, f_r.data_ptr(), fs_r.data_ptr(),
                                            f_c.data_ptr(), fs_c.data_ptr(), st), "rowcol")
    torch.cuda.synchronize()
    assert torch.equal(f_r, q_r) and torch.equal(f_c, q_c)
    assert torch.equal(fs_c, s_c)
    # row scales: compare the entries of real rows (the row kernel leaves other positions untouched as well)
    r, c = np.meshgrid(np.arange(rows), np.arange(cols // 32), indexing="ij")
    idx = Q.blocked_scale_offset(r, c, ra)
    np.testing.assert_array_equal(fs_r.cpu().numpy()[idx], s_r.cpu().numpy()[idx])


@pytest.mark.parametrize("rows,cols,cap", [(96, 512, 128), (200, 1536, 256)])
def test_mxfp8_rowcol_with_gather_and_with_swiglu_equal_the_staged_forms(rows, cols, cap):
    """The quantiser that pulls rows through a pointer table, and the one that applies SwiGLU to h1 first, give the
    bytes of gather -> quantise and SwiGLU -> quantise run as separate kernels."""
    nat = _nat()
    st = nat.stream_ptr()
    cnt = torch.tensor([rows], dtype=torch.int32, device=DEV)
    ra, ca = (cols // 32 + 3) // 4, ((cap + 31) // 32 + 3) // 4
    n_rs, n_cs = (cap + 127) // 128 * 128 * ra * 4, (cols + 127) // 128 * 128 * ca * 4

    def outputs():
        return (torch.zeros(cap, cols, dtype=torch.uint8, device=DEV), torch.zeros(n_rs, dtype=torch.uint8, device=DEV),
                torch.zeros(cap, cols, dtype=torch.uint8, device=DEV), torch.zeros(n_cs, dtype=torch.uint8, device=DEV))

    # --- gather: a permutation of source rows with every seventh pointer null
    src = _data(rows, cols, rows + 11, specials=False).to(DEV)
    perm = torch.randperm(rows, generator=torch.Generator().manual_seed(rows))
    ptrs = torch.tensor([0 if i % 7 == 3 else src.data_ptr() + int(perm[i]) * cols * 2 for i in range(rows)],
                        dtype=torch.int64, device=DEV)
    dense = src[perm.to(DEV)].clone()
    dense[torch.arange(rows, device=DEV) % 7 == 3] = 0
    want = outputs()
    nat.check(nat.lib.dm_quant_mxfp8_rowcol(dense.data_ptr(), cnt.data_ptr(), cap, cols, want[0].data_ptr(),
                                            want[1].data_ptr(), want[2].data_ptr(), want[3].data_ptr(), st), "rowcol")
    got = outputs()
    nat.check(nat.lib.dm_quant_mxfp8_rowcol_gather(ptrs.data_ptr(), cnt.data_ptr(), cap, cols, got[0].data_ptr(),
                                                   got[1].data_ptr(), got[2].data_ptr(), got[3].data_ptr(), st), "gather")
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert torch.equal(g, w)

    # --- SwiGLU (plain and clamped) of h1 = [gate | up]
    for clamped in (0, 1):
        h1 = (torch.randn(rows, 2 * cols, generator=torch.Generator().manual_seed(5 + clamped)) * 3).bfloat16().to(DEV)
        h2 = torch.zeros(rows, cols, dtype=torch.bfloat16, device=DEV)
        nat.check(nat.lib.dm_swiglu_fwd(h1.data_ptr(), None, h2.data_ptr(), None, cnt.data_ptr(), rows, cols, clamped, 1.702,
                                        7.0, None, 0.0, None, st), "swiglu")
        want = outputs()
        nat.check(nat.lib.dm_quant_mxfp8_rowcol(h2.data_ptr(), cnt.data_ptr(), cap, cols, want[0].data_ptr(),
                                                want[1].data_ptr(), want[2].data_ptr(), want[3].data_ptr(), st), "rowcol")
        got = outputs()
        nat.check(nat.lib.dm_swiglu_fwd_quant_mxfp8_rowcol(h1.data_ptr(), cnt.data_ptr(), cap, cols, clamped, 1.702, 7.0,
                                                           got[0].data_ptr(), got[1].data_ptr(), got[2].data_ptr(),
                                                           got[3].data_ptr(), st), "swiglu+quant")
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g, w)


@pytest.mark.parametrize("rows,F,cap,clamped", [(96, 512, 128, 0), (200, 1536, 256, 1), (70, 96, 128, 0)])
def test_swiglu_backward_fused_into_the_quantiser_equals_the_staged_form(rows, F, cap, clamped):
    """dm_swiglu_bwd_quant_mxfp8 gives the bytes of dm_swiglu_bwd followed by the row+column quantiser, and leaves
    out the copy that is not asked for."""
    nat = _nat()
    st = nat.stream_ptr()
    cnt = torch.tensor([rows], dtype=torch.int32, device=DEV)
    C = 2 * F
    ra, ca = (C // 32 + 3) // 4, ((cap + 31) // 32 + 3) // 4
    n_rs, n_cs = (cap + 127) // 128 * 128 * ra * 4, (C + 127) // 128 * 128 * ca * 4

    def outputs():
        return (torch.zeros(cap, C, dtype=torch.uint8, device=DEV), torch.zeros(n_rs, dtype=torch.uint8, device=DEV),
                torch.zeros(cap, C, dtype=torch.uint8, device=DEV), torch.zeros(n_cs, dtype=torch.uint8, device=DEV))

    g = torch.Generator().manual_seed(31 + rows)
    h1 = (torch.randn(rows, C, generator=g) * 4).bfloat16().to(DEV)
    dz = (torch.randn(rows, F, generator=g) * torch.logspace(-3, 2, rows)[:, None]).bfloat16().to(DEV)
    dh1 = torch.zeros(rows, C, dtype=torch.bfloat16, device=DEV)
    nat.check(nat.lib.dm_swiglu_bwd(h1.data_ptr(), None, dz.data_ptr(), None, dh1.data_ptr(), None, cnt.data_ptr(), rows, F,
                                    clamped, 1.702, 7.0, st), "swiglu_bwd")
    want = outputs()
    nat.check(nat.lib.dm_quant_mxfp8_rowcol(dh1.data_ptr(), cnt.data_ptr(), cap, C, want[0].data_ptr(), want[1].data_ptr(),
                                            want[2].data_ptr(), want[3].data_ptr(), st), "rowcol")
    got = outputs()
    nat.check(nat.lib.dm_swiglu_bwd_quant_mxfp8(h1.data_ptr(), dz.data_ptr(), cnt.data_ptr(), cap, F, clamped, 1.702, 7.0,
                                                got[0].data_ptr(), got[1].data_ptr(), got[2].data_ptr(), got[3].data_ptr(),
                                                st), "fused")
    only_row, only_col = outputs(), outputs()
    nat.check(nat.lib.dm_swiglu_bwd_quant_mxfp8(h1.data_ptr(), dz.data_ptr(), cnt.data_ptr(), cap, F, clamped, 1.702, 7.0,
                                                only_row[0].data_ptr(), only_row[1].data_ptr(), None, None, st), "row only")
    nat.check(nat.lib.dm_swiglu_bwd_quant_mxfp8(h1.data_ptr(), dz.data_ptr(), cnt.data_ptr(), cap, F, clamped, 1.702, 7.0,
                                                None, None, only_col[2].data_ptr(), only_col[3].data_ptr(), st), "col only")
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert torch.equal(only_row[0], want[0]) and torch.equal(only_row[1], want[1]) and not only_row[2].any()
    assert torch.equal(only_col[2], want[2]) and torch.equal(only_col[3], want[3]) and not only_col[0].any()


@pytest.mark.parametrize("rows,cols", [(96, 2048), (40, 7168)])
def test_nvfp4_token_live_rows_only(rows, cols):
    """dm_quant_nvfp4_token_live quantises the rows whose table entry is non-zero exactly as the plain call does
    and leaves the others untouched."""
    nat = _nat()
    st = nat.stream_ptr()
    x = _data(rows, cols, rows + 5, specials=False).to(DEV)
    live = torch.tensor([0 if r % 3 == 1 else 1000 + r for r in range(rows)], dtype=torch.int64, device=DEV)

    def outputs(fill):
        return (torch.full((rows, cols // 2), fill, dtype=torch.uint8, device=DEV),
                torch.full((rows, cols // 16), fill, dtype=torch.uint8, device=DEV),
                torch.full((rows,), float(fill), dtype=torch.float32, device=DEV))

    want, got = outputs(0), outputs(0xAB)
    nat.check(nat.lib.dm_quant_nvfp4_token(x.data_ptr(), None, rows, cols, want[0].data_ptr(), cols // 2, want[1].data_ptr(),
                                           cols // 16, 0, want[2].data_ptr(), 4, st), "plain")
    nat.check(nat.lib.dm_quant_nvfp4_token_live(live.data_ptr(), x.data_ptr(), None, rows, cols, got[0].data_ptr(), cols // 2,
                                                got[1].data_ptr(), cols // 16, 0, got[2].data_ptr(), 4, st), "live")
    torch.cuda.synchronize()
    keep = live != 0
    for g, w in zip(got, want):
        assert torch.equal(g[keep], w[keep])
    assert bool((got[0][~keep] == 0xAB).all()) and bool((got[1][~keep] == 0xAB).all())
    assert bool((got[2][~keep] == float(0xAB)).all())


@pytest.mark.parametrize("rows,cols,gather,offset", [(1, 32, 0, 0), (127, 96, 1, 0), (128, 128, 0, 0), (129, 160, 1, 0),
                                                     (261, 384, 0, 2), (300, 288, 1, 2), (384, 1056, 1, 0)])
def test_mxfp8_rowcol_tile_edges_against_the_oracle(rows, cols, gather, offset):
    """Both copies and both scale sets at the edges of the 128 x 128 tiles (partial rows, partial 32-row blocks, partial
    column tiles), with blocks that are zero, infinite, NaN, subnormal or exactly 448 * 2^k, null row pointers, and
    output buffers that are only 2-byte aligned.  Integer results: equal."""
    nat = _nat()
    x = _data(rows, cols, 7 * rows + cols)
    x[:, 5] = 0
    x[rows // 2, :] = 448.0 * 2.0 ** -6  # amax / 448 is a power of two: the scale must not round up
    x[rows - 1, : min(32, cols)] = 2.0 ** -133  # subnormal bf16
    cap = rows + 3
    cnt = torch.tensor([rows], dtype=torch.int32, device=DEV)
    ra, ca = (cols // 32 + 3) // 4, ((cap + 31) // 32 + 3) // 4
    n_rs, n_cs = (cap + 127) // 128 * 128 * ra * 4, (cols + 127) // 128 * 128 * ca * 4
    qr = torch.zeros(cap * cols, dtype=torch.uint8, device=DEV)
    sr = torch.full((n_rs + 16,), 0xEE, dtype=torch.uint8, device=DEV)[offset: offset + n_rs]
    qc = torch.zeros(cap * cols + 16, dtype=torch.uint8, device=DEV)[offset: offset + cap * cols]
    sc = torch.full((n_cs + 16,), 0xEE, dtype=torch.uint8, device=DEV)[offset: offset + n_cs]
    xd = x.to(DEV)
    out = (qr.data_ptr(), sr.data_ptr(), qc.data_ptr(), sc.data_ptr())
    if gather:
        null = torch.arange(rows) % 5 == 2
        ptrs = torch.where(null, 0, xd.data_ptr() + torch.arange(rows) * cols * 2).to(DEV)
        x[null] = 0
        nat.check(nat.lib.dm_quant_mxfp8_rowcol_gather(ptrs.data_ptr(), cnt.data_ptr(), cap, cols, *out, nat.stream_ptr()), "gather")
    else:
        nat.check(nat.lib.dm_quant_mxfp8_rowcol(xd.data_ptr(), cnt.data_ptr(), cap, cols, *out, nat.stream_ptr()), "rowcol")
    torch.cuda.synchronize()

    def same(got, want, scales):  # data of non-finite blocks is NaN of either sign
        finite = scales != 255
        np.testing.assert_array_equal(got[finite], want[finite])
        assert ((got[~finite] & 0x7F) == 0x7F).all()

    rq, rs = Q.mxfp8_row(x)
    r, c = np.meshgrid(np.arange(rows), np.arange(cols // 32), indexing="ij")
    np.testing.assert_array_equal(sr.cpu().numpy()[Q.blocked_scale_offset(r, c, ra)], rs)
    same(qr.cpu().numpy().reshape(cap, cols)[:rows], rq, np.repeat(rs, 32, axis=1))
    cq, cs = Q.mxfp8_col(x)
    c, b = np.meshgrid(np.arange(cols), np.arange((rows + 31) // 32), indexing="ij")
    np.testing.assert_array_equal(sc.cpu().numpy()[Q.blocked_scale_offset(c, b, ca)], cs)
    same(qc.cpu().numpy().reshape(cap, cols)[:rows], cq, np.repeat(cs.T, 32, axis=0)[:rows])
    # nothing outside the matrix was written
    assert int(qr.view(cap, cols)[rows:].sum()) == 0 and int(qc.view(cap, cols)[rows:].sum()) == 0
    assert int((sr.cpu() == 0xEE).sum()) >= n_rs - rs.size
    assert int((sc.cpu() == 0xEE).sum()) >= n_cs - cs.size


@pytest.mark.parametrize("rows,cols", [(70, 16), (33, 512), (40, 528), (35, 1040), (21, 2064), (12, 4112), (9, 8192), (6, 8208)])
def test_nvfp4_token_row_lengths_at_the_limits_of_the_register_forms(rows, cols):
    """The warp-per-row (up to 2048 elements), CTA-per-row (8192) and two-pass forms, with an all-zero row and blocks that
    hold infinities; packed bytes, block scales and inverse row scales equal the oracle's.  A NaN leaves the row's scale
    to the other elements."""
    nat = _nat()
    x = _data(rows, cols, rows + cols, specials=False)
    x[1] = 0
    rp, rs, rinv = Q.nvfp4_token_rows(x)
    xn = x.clone()
    xn[2, cols - 1] = float("nan")
    amax = torch.nan_to_num(xn[2].float(), nan=0.0).abs().max()

    def run(t):
        q = torch.zeros(rows, cols // 2, dtype=torch.uint8, device=DEV)
        s = torch.zeros(rows, cols // 16, dtype=torch.uint8, device=DEV)
        inv = torch.zeros(rows, dtype=torch.float32, device=DEV)
        nat.check(nat.lib.dm_quant_nvfp4_token(t.to(DEV).data_ptr(), None, rows, cols, q.data_ptr(), cols // 2, s.data_ptr(),
                                               cols // 16, 0, inv.data_ptr(), 4, nat.stream_ptr()), "nvfp4_token")
        torch.cuda.synchronize()
        return q.cpu().numpy(), s.cpu().numpy(), inv.cpu().numpy()

    q, s, inv = run(x)
    np.testing.assert_array_equal(inv.view(np.uint32), rinv.view(np.uint32))
    np.testing.assert_array_equal(s, rs)
    np.testing.assert_array_equal(q, rp)
    q, s, inv = run(xn)
    assert abs(inv[2] * 2688.0 / float(amax) - 1.0) < 1e-6
    others = np.arange(rows) != 2
    np.testing.assert_array_equal(q[others], rp[others])
    np.testing.assert_array_equal(s[others], rs[others])


@pytest.mark.parametrize("rows,q_bytes,scale_cols,has_inv", [(1, 16, 4, 0), (128, 2064, 132, 1), (200, 2816, 88, 0), (384, 3584, 448, 1)])
def test_gather_packed_rows_unpacks_every_row_and_atom(rows, q_bytes, scale_cols, has_inv):
    """Whole 128-row blocks (written sector by sector) and a partial last one, atom counts around a warp's 32, null
    pointers as rows of zeros; plain copies of bytes: equal."""
    nat = _nat()
    stride = (q_bytes + scale_cols + 4 * has_inv + 15) // 16 * 16
    g = torch.Generator().manual_seed(rows)
    packed = torch.randint(0, 256, (rows, stride), dtype=torch.uint8, generator=g)
    perm = torch.randperm(rows, generator=g)
    null = torch.arange(rows) % 6 == 4
    src = packed.to(DEV)
    ptrs = torch.where(null, 0, src.data_ptr() + perm * stride).to(DEV)
    cap = rows + 5
    atoms = scale_cols // 4
    q = torch.full((cap, q_bytes), 0xEE, dtype=torch.uint8, device=DEV)
    sf = torch.full(((cap + 127) // 128 * 128 * scale_cols,), 0xEE, dtype=torch.uint8, device=DEV)
    inv = torch.full((cap, 4), 0xEE, dtype=torch.uint8, device=DEV)
    cnt = torch.tensor([rows], dtype=torch.int32, device=DEV)
    op = lambda t: nat.Operand(t.data_ptr(), t.numel(), None)  # noqa: E731
    ptrs_cap = torch.cat([ptrs, torch.zeros(5, dtype=torch.int64, device=DEV)])
    nat.check(nat.lib.dm_gather_packed_rows(ptrs_cap.data_ptr(), cnt.data_ptr(), cap, q_bytes, scale_cols, has_inv, op(q), op(sf),
                                            op(inv) if has_inv else nat.Operand(None, 0, None), None, nat.stream_ptr()), "gather")
    torch.cuda.synchronize()
    want = packed[perm].clone()
    want[null] = 0
    np.testing.assert_array_equal(q.cpu().numpy()[:rows], want[:, :q_bytes].numpy())
    r, c = np.meshgrid(np.arange(rows), np.arange(scale_cols), indexing="ij")
    got = sf.cpu().numpy()
    np.testing.assert_array_equal(got[Q.blocked_scale_offset(r, c, atoms)], want[:, q_bytes: q_bytes + scale_cols].numpy())
    if has_inv:
        np.testing.assert_array_equal(inv.cpu().numpy()[:rows], want[:, q_bytes + scale_cols: q_bytes + scale_cols + 4].numpy())
    assert bool((q[rows:] == 0xEE).all())
    assert int((got == 0xEE).sum()) >= got.size - rows * scale_cols


@pytest.mark.parametrize("rows,cols", [(4, 32), (37, 1056), (64, 2816)])
def test_mxfp8_row_live_rows_only(rows, cols):
    """dm_quant_mxfp8_row_live quantises the rows whose table entry is non-zero exactly as the plain call does and leaves
    the others untouched; the plain call equals the oracle on the same rows."""
    nat = _nat()
    st = nat.stream_ptr()
    x = _data(rows, cols, rows + 5)
    xd = x.to(DEV)
    live = torch.tensor([0 if r % 3 == 1 else 1000 + r for r in range(rows)], dtype=torch.int64, device=DEV)
    want, got = ((torch.full((rows, cols), 0xAB, dtype=torch.uint8, device=DEV),
                  torch.full((rows, cols // 32), 0xAB, dtype=torch.uint8, device=DEV)) for _ in range(2))
    nat.check(nat.lib.dm_quant_mxfp8_row(xd.data_ptr(), None, rows, cols, want[0].data_ptr(), 0, want[1].data_ptr(), 0, 0, st), "plain")
    nat.check(nat.lib.dm_quant_mxfp8_row_live(live.data_ptr(), xd.data_ptr(), None, rows, cols, got[0].data_ptr(), 0,
                                              got[1].data_ptr(), 0, 0, st), "live")
    torch.cuda.synchronize()
    rq, rs = Q.mxfp8_row(x)
    np.testing.assert_array_equal(want[1].cpu().numpy(), rs)
    finite = np.repeat(rs != 255, 32, axis=1)
    np.testing.assert_array_equal(want[0].cpu().numpy()[finite], rq[finite])
    keep = live != 0
    for g, w in zip(got, want):
        assert torch.equal(g[keep], w[keep]) and bool((g[~keep] == 0xAB).all())


@pytest.mark.parametrize("rows,cols", [(1, 32), (130, 160)])
def test_mxfp8_gather_from_a_table_that_is_only_8_byte_aligned(rows, cols):
    """A pointer table may start at any 8-byte address; null pointers, rows past the end and columns past the matrix read
    nothing.  Same bytes as from a table on 16 bytes."""
    nat = _nat()
    x = _data(rows, cols, 3 * rows + cols, specials=False).to(DEV)
    ptrs = torch.where(torch.arange(rows) % 4 == 3, 0, x.data_ptr() + torch.arange(rows) * cols * 2)
    ra, ca = (cols // 32 + 3) // 4, ((rows + 31) // 32 + 3) // 4
    got = []
    for shift in (0, 1):
        table = torch.zeros(rows + 2, dtype=torch.int64, device=DEV)
        table[shift:shift + rows] = ptrs.to(DEV)
        assert table[shift:].data_ptr() % 16 == 8 * shift
        out = [torch.zeros(n, dtype=torch.uint8, device=DEV)
               for n in (rows * cols, (rows + 127) // 128 * 128 * ra * 4, rows * cols, (cols + 127) // 128 * 128 * ca * 4)]
        nat.check(nat.lib.dm_quant_mxfp8_rowcol_gather(table[shift:].data_ptr(), None, rows, cols, *[t.data_ptr() for t in out],
                                                       nat.stream_ptr()), "gather")
        torch.cuda.synchronize()
        got.append(out)
    assert all(torch.equal(a, b) for a, b in zip(*got)) and bool(got[0][0].any())


@pytest.mark.parametrize("experts,n,k", [(1, 128, 128), (3, 256, 384), (2, 640, 128), (2, 128, 1152)])
def test_mxfp8_tile32_forms_agree(experts, n, k):
    """Aligned weights take the 128 x 128 form, the same weights two bytes further the slab form: equal bytes, with zero tiles,
    infinities, NaNs and subnormals among the values."""
    nat = _nat()
    g = torch.Generator().manual_seed(n + k)
    w = (torch.randn(experts, n, k, generator=g) * torch.exp2(torch.randint(-140, 120, (experts, n // 32, 1, k // 32, 1), generator=g)
         .float()).expand(-1, -1, 32, -1, 32).reshape(experts, n, k)).bfloat16()
    w[0, :32, :32] = 0
    w[0, 5, 40] = float("inf")
    w[-1, 100, 127] = float("nan")
    flat = w.reshape(-1)
    shifted = torch.zeros(flat.numel() + 1, dtype=torch.bfloat16, device=DEV)
    shifted[1:] = flat.to(DEV)
    aligned = flat.to(DEV)
    out = []
    for src in (aligned.data_ptr(), shifted.data_ptr() + 2):
        q = torch.zeros(experts * n * k, dtype=torch.uint8, device=DEV)
        s0 = torch.zeros(experts * n * (k // 32), dtype=torch.uint8, device=DEV)
        s1 = torch.zeros(experts * k * (n // 32), dtype=torch.uint8, device=DEV)
        nat.check(nat.lib.dm_quant_mxfp8_tile32(src, experts, n, k, q.data_ptr(), s0.data_ptr(), s1.data_ptr(), 1,
                                                nat.stream_ptr()), "tile32")
        out.append((q, s0, s1))
    torch.cuda.synchronize()
    for a, b in zip(*out):
        assert torch.equal(a, b)
