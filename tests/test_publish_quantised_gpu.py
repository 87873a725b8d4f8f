"""The launch that publishes an inference call (quantised tokens and expert ids together) against the launches it stands for, and the
gather that leaves padding rows alone against the one that zeroes them: the same bytes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _geometry(fmt, D):
    q, s = (D, D // 32) if fmt == 0 else (D // 2, D // 16)
    s = (s + 3) // 4 * 4
    return q, s, (q + s + (4 if fmt else 0) + 15) // 16 * 16


# warp-sized rows, rows of a block, rows that no block holds (NVFP4: read twice)
@pytest.mark.parametrize("fmt,D", [(0, 128), (0, 2816), (1, 256), (1, 2048), (1, 4096), (1, 7168), (1, 8448)])
@pytest.mark.parametrize("T,K,ids_dtype", [(1, 1, torch.int64), (33, 5, torch.int32), (700, 8, torch.int64)])
def test_one_launch_publishes_what_two_did(fmt, D, T, K, ids_dtype):
    from dist_moe_b200 import _native as nat

    E, st = 32, nat.stream_ptr()
    torch.manual_seed(T + D)
    q, s, stride = _geometry(fmt, D)
    x = torch.randn(T, D, device=DEV).bfloat16()
    ids = torch.randint(-1, E, (T, K), device=DEV).to(ids_dtype)
    ids[T // 2, 0] = E  # reported by both
    rows = [torch.full((T * stride,), 0xAB, dtype=torch.uint8, device=DEV) for _ in range(2)]
    routing = [torch.full((128 + 2 * T * K + 64,), 0xAB, dtype=torch.uint8, device=DEV) for _ in range(2)]
    status = [torch.zeros(8, dtype=torch.int32, device=DEV) for _ in range(2)]
    at = rows[0].data_ptr()
    if fmt:
        nat.check(nat.lib.dm_quant_nvfp4_token(x.data_ptr(), None, T, D, at, stride, at + q, stride, 0, at + q + s, stride, st), "q")
    else:
        nat.check(nat.lib.dm_quant_mxfp8_row(x.data_ptr(), None, T, D, at, stride, at + q, stride, 0, st), "q")
    nat.check(nat.lib.dm_publish(None, ids.data_ptr(), int(ids_dtype is torch.int64), None, routing[0].data_ptr(), T, 0, K, E, 1,
                                 status[0].data_ptr(), st), "publish")
    nat.check(nat.lib.dm_publish_quantised(fmt, x.data_ptr(), ids.data_ptr(), int(ids_dtype is torch.int64), rows[1].data_ptr(), stride,
                                           q, s, routing[1].data_ptr(), T, D, K, E, 1, status[1].data_ptr(), st), "one launch")
    torch.cuda.synchronize()
    assert torch.equal(rows[0], rows[1]) and torch.equal(routing[0], routing[1])
    assert status[0][0].item() != 0 and torch.equal(status[0][:1], status[1][:1])


@pytest.mark.parametrize("has_inv", [0, 1])
@pytest.mark.parametrize("counts", [[1, 0, 33, 128], [130, 2], [128]])
@pytest.mark.parametrize("q_bytes", [128, 2176])
def test_live_gather_leaves_padding_rows(has_inv, counts, q_bytes):
    from dist_moe_b200 import _native as nat

    torch.manual_seed(q_bytes)
    s_cols = q_bytes // 32 if not has_inv else q_bytes // 8
    s_cols = (s_cols + 3) // 4 * 4
    stride = (q_bytes + s_cols + 4 * has_inv + 15) // 16 * 16
    src = torch.randint(0, 256, (300, stride), dtype=torch.uint8, device=DEV)
    live, rows = [], 0
    for c in counts:
        live += range(rows, rows + c)
        rows += (c + 127) // 128 * 128
    live = torch.tensor(live, device=DEV)
    ptrs = torch.zeros(rows, dtype=torch.int64, device=DEV)
    ptrs[live] = src.data_ptr() + torch.randint(0, 300, (len(live),), device=DEV) * stride
    num = torch.tensor([rows], dtype=torch.int32, device=DEV)
    atoms = (s_cols + 3) // 4
    got = {}
    for name in ("dm_gather_packed_rows", "dm_gather_packed_rows_live"):
        bufs = [torch.full((n,), 0xAB, dtype=torch.uint8, device=DEV) for n in (rows * q_bytes, rows // 128 * atoms * 512, rows * 4)]
        op = lambda t: nat.Operand(t.data_ptr(), t.numel(), None)  # noqa: E731
        nat.check(getattr(nat.lib, name)(ptrs.data_ptr(), num.data_ptr(), rows, q_bytes, s_cols, has_inv, op(bufs[0]), op(bufs[1]),
                                         op(bufs[2]), None, nat.stream_ptr()), name)
        torch.cuda.synchronize()
        got[name] = bufs
    whole, part = got.values()
    # byte (row % 32) * 16 + (row // 32 % 4) * 4 + column of an atom of 128 rows x 4 columns
    scales = [b[1].view(rows // 128, atoms, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(rows, atoms * 4) for b in (whole, part)]
    for a, b in ((whole[0].view(rows, -1), part[0].view(rows, -1)), scales, (whole[2].view(rows, -1), part[2].view(rows, -1))):
        assert torch.equal(a[live], b[live])
    dead = torch.ones(rows, dtype=torch.bool, device=DEV)
    dead[live] = False
    assert bool((part[0].view(rows, -1)[dead] == 0xAB).all()) and bool((whole[0].view(rows, -1)[dead] == 0).all())
