"""Row + column quantiser with two scales worked out at a time, over every bf16 pattern: finite blocks, blocks that an infinity or a NaN
makes non-finite next to finite ones in the same lane, and all exponents.  The row copy against the row quantiser (one scale at a time),
the column copy against the slab form (fp32 arithmetic), byte for byte."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [256, 131])  # whole tiles, and a last tile of three rows
@pytest.mark.parametrize("kind", ["finite", "mixed", "exponents"])
def test_every_pattern(kind, rows):
    from dist_moe_b200 import _native as nat

    dev, C, st = torch.device("cuda", 0), 256, nat.stream_ptr()
    g = torch.Generator().manual_seed(5)
    bits = torch.arange(65536)[torch.randperm(65536, generator=g)].reshape(256, C)
    if kind == "finite":
        bits[(bits & 0x7F80) == 0x7F80] &= 0x3FFF
    elif kind == "mixed":  # few non-finite values, so that most blocks have none
        bad = (bits & 0x7F80) == 0x7F80
        bits[bad & (torch.rand(bits.shape, generator=g) > 0.05)] &= 0x3FFF
    else:  # neighbouring values of one magnitude: scales of every size
        bits = (torch.arange(256)[:, None] // 32 * 32 + torch.arange(C)[None, :] // 32 * 4) % 255 * 128 + bits % 128
    bits = bits[:rows]
    x = bits.to(torch.int32).to(torch.int16).view(torch.bfloat16).contiguous().to(dev)
    if kind == "exponents":
        assert not bool(torch.isnan(x.float()).any())
    atoms = lambda n: (n + 3) // 4  # noqa: E731
    new = lambda n: torch.zeros(n, dtype=torch.uint8, device=dev)  # noqa: E731
    cols_of_rows = (rows + 31) // 32
    q_row, q_col, want_row, want_col = (new(rows * C) for _ in range(4))
    s_row, want_s_row = (new((rows + 127) // 128 * 128 * atoms(C // 32) * 4) for _ in range(2))
    s_col, want_s_col = (new(C * atoms(cols_of_rows) * 4) for _ in range(2))
    nat.check(nat.lib.dm_quant_mxfp8_rowcol(x.data_ptr(), None, rows, C, q_row.data_ptr(), s_row.data_ptr(), q_col.data_ptr(),
                                            s_col.data_ptr(), st), "rowcol")
    nat.check(nat.lib.dm_quant_mxfp8_row(x.data_ptr(), None, rows, C, want_row.data_ptr(), 0, want_s_row.data_ptr(), 0, 1, st), "row")
    # a source that does not start on 16 bytes takes the slab form
    shifted = torch.empty(rows * C + 4, dtype=torch.bfloat16, device=dev)[4:]
    shifted.copy_(x.reshape(-1))
    nat.check(nat.lib.dm_quant_mxfp8_col(shifted.data_ptr(), None, rows, C, want_col.data_ptr(), want_s_col.data_ptr(), 1, st), "col")
    torch.cuda.synchronize()
    assert torch.equal(q_row, want_row) and torch.equal(s_row, want_s_row)
    assert torch.equal(q_col, want_col) and torch.equal(s_col, want_s_col)
