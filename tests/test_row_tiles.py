"""Row tiles of the BF16 forward / input-gradient GEMM and the gathered row blocks each tile waits for (CPU).

The kernel's own arithmetic (csrc/row_tiles.cuh) is compiled for the host and walked the way a CTA pair walks its tiles.
"""

import ctypes
import random
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "dist_moe_b200" / "csrc"
BLOCK = 128

HARNESS = r"""
#include "row_tiles.cuh"
#include <vector>
using namespace dm;
// Tiles of CTA pair `first` of `step`, in its order: eight ints each.
extern "C" int walk(const int* off, int experts, int m_pairs, int first, int step, int* out, int capacity) {
  std::vector<int> start(experts + 1);
  std::vector<uint16_t> per(experts);
  for (int e = 0; e < experts; ++e) {
    const int rows = off[e + 1] - off[e];
    per[e] = static_cast<uint16_t>(rw_rows_per_tile(rows));
    start[e + 1] = start[e] + rw_row_tiles(rows) * m_pairs;
  }
  int e = 0, n = 0;
  for (int tile = first; tile < start[experts]; tile += step, ++n) {
    if (n == capacity) return -1;
    const RowsTile t = rw_decode(tile, e, start.data(), off, per.data());
    const RowsBlocks b = rw_tile_blocks(t, off[experts]);
    const int v[8] = {t.e, t.pair, t.row0, t.rows, t.n, b.first, b.last, 2 * rw_box_rows(rw_box_index(t.n))};
    for (int i = 0; i < 8; ++i) out[8 * n + i] = v[i];
  }
  return n;
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    folder = tmp_path_factory.mktemp("row_tiles")
    (folder / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-x", "c++", str(folder / "harness.cpp"), f"-I{CSRC}",
                    "-o", str(folder / "harness.so")], check=True)
    lib = ctypes.CDLL(str(folder / "harness.so"))

    def call(counts, n, pair, pairs):
        off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
        m_pairs = (n + 255) // 256
        out = np.zeros((int((-(-np.array(counts) // 256)).sum()) * m_pairs + 1, 8), dtype=np.int32)
        got = lib.walk(off.ctypes.data_as(ctypes.c_void_p), len(counts), m_pairs, pair, pairs,
                       out.ctypes.data_as(ctypes.c_void_p), len(out))
        assert got >= 0
        return out[:got]

    return call


def _scenarios():
    yield [3072] * 8, 2816, 74          # long experts: a pair's second tile lies before its first one
    yield [2048] * 4, 3072, 74
    yield [1], 64, 1
    yield [0, 257, 0, 2049, 1, 255, 256, 4095], 1408, 3
    rng = random.Random(3)
    for _ in range(60):
        experts = rng.randint(1, 24)
        counts = [rng.choice([0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, rng.randint(0, 4000)]) for _ in range(experts)]
        yield counts, 8 * rng.randint(8, 400), rng.randint(1, 74)


def test_tiles_cover_every_row_and_wait_for_every_block_they_use(walk):
    for counts, n, pairs in _scenarios():
        m_pairs = (n + 255) // 256
        seen = np.zeros((sum(counts), m_pairs), dtype=np.int32)
        off = np.concatenate([[0], np.cumsum(counts)])
        for pair in range(pairs):
            for e, col, row0, rows, tile_n, first, last, box in walk(counts, n, pair, pairs):
                assert off[e] <= row0 and 0 < rows and row0 + rows <= off[e + 1]
                assert rows <= tile_n <= 256 and tile_n % 32 == 0 and tile_n <= box
                seen[row0:row0 + rows, col] += 1
                # the blocks the tile waits for hold all the rows it uses, exist, and fit a lane each
                assert first * BLOCK <= row0 and row0 + rows <= (last + 1) * BLOCK
                assert last * BLOCK < sum(counts) and last - first < 32
        assert (seen == 1).all()


@pytest.mark.parametrize("counts,n", [([3072] * 8, 2816), ([2048] * 4, 3072)])
def test_a_high_water_mark_would_leave_blocks_unchecked(walk, counts, n):
    """Why every tile waits for its own blocks: taking everything below the highest block waited for so far as landed
    skips blocks that only other CTAs have looked at."""
    skipped = 0
    for pair in range(74):
        mark, checked = 0, set()
        for _, _, _, _, _, first, last, _ in walk(counts, n, pair, 74):
            if last >= mark:
                checked.update(range(max(mark, first), last + 1))
                mark = last + 1
            skipped += len(set(range(first, last + 1)) - checked)
    assert skipped > 0


def test_pairs_that_take_tiles(tmp_path):
    """Even rounds: no more rounds than with all pairs, every pair with tiles in all of them but the last; all pairs where rounds
    do not matter (one round, large tiles), and, where the epilogue counts, where two or three rounds fill more than half of the last."""
    (tmp_path / "p.cpp").write_text('#include "row_tiles.cuh"\nextern "C" int pairs(int t, int w, int r, int l, bool h) '
                                    '{ return dm::balanced_pairs(t, w, r, l, h); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(tmp_path / "p.so"), str(tmp_path / "p.cpp")],
                   check=True)
    pairs = ctypes.CDLL(str(tmp_path / "p.so")).pairs
    pairs.argtypes = [ctypes.c_int] * 4 + [ctypes.c_bool]
    for workers in (1, 3, 74):
        for tiles in range(0, 12 * workers + 2):
            rounds = -(-tiles // workers)
            assert pairs(tiles, workers, 65, 64, False) == workers
            even = pairs(tiles, workers, 64, 64, False)
            assert even == workers if rounds <= 1 else even <= workers and (rounds - 1) * even < tiles <= rounds * even
            heavy = pairs(tiles, workers, 64, 64, True)
            last = tiles - (rounds - 1) * workers
            assert heavy == (workers if 2 <= rounds <= 3 and 2 * last > workers else even)
    # measured: 132 tiles (58 in the second round) and 198 (50 in the third) lose by even rounds, 154 (6), 242 and 264 gain
    assert [pairs(t, 74, 32, 32, True) for t in (132, 198, 154, 242, 264)] == [74, 74, 52, 61, 66]
