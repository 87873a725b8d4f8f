"""Rows that the block-scaled GEMMs work on (CPU): the arithmetic of csrc/row_tiles.cuh, compiled for the host."""

import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "dist_moe_b200" / "csrc"

HARNESS = r"""
#include "row_tiles.cuh"
using namespace dm;
extern "C" int group_rows(int off, int next, int count) { return bs_group_rows(off, next, count); }
// Tiles of one expert of `rows` rows at a group's start: first row and rows (the MMA's N) of each, and the size of its box.
extern "C" int tiles(int rows, int* out) {
  const int nt = rw_row_tiles(rows), per = bs_rows_per_tile(rows);
  for (int i = 0; i < nt; ++i) {
    const int left = rows - i * per, mine = left < per ? left : per;
    out[3 * i] = i * per;
    out[3 * i + 1] = mine > 0 ? (mine + 31) & ~31 : 32;
    out[3 * i + 2] = 2 * rw_box_rows(rw_box_index(per));
  }
  return nt;
}
extern "C" int tile_atoms(int n_max) { return bs_tile_atoms(n_max); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    folder = tmp_path_factory.mktemp("bs_row_tiles")
    (folder / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", str(folder / "harness.cpp"), f"-I{CSRC}",
                    "-o", str(folder / "harness.so")], check=True)
    return ctypes.CDLL(str(folder / "harness.so"))


def test_a_group_that_starts_inside_a_scale_atom_is_left_out(lib):
    """Its tiles would name odd TMEM columns as their scale address, on which the GPU faults."""
    for off in range(0, 513):
        for rows in (1, 31, 32, 33, 128, 200, 700):
            got = lib.group_rows(off, off + rows, 1 << 30)
            assert got == (rows if off % 128 == 0 else 0)


def test_rows_stay_inside_the_group(lib):
    for room in (0, 1, 128, 256):
        for count in (-5, 0, 1, 127, 128, 129, 1000):
            assert lib.group_rows(256, 256 + room, count) == max(0, min(room, count))
    assert lib.group_rows(256, 128, 40) == 0  # the end of the rows lies before the group


def test_tiles_touch_no_more_scale_atoms_than_a_stage_holds(lib):
    out = (ctypes.c_int * 300)()
    for rows in range(1, 20000):
        n = lib.tiles(rows, out)
        covered = 0
        for i in range(n):
            start, size, box = out[3 * i:3 * i + 3]
            assert start == covered and start % 64 == 0 and size <= box  # an even scale column, rows without a gap
            assert (start + size - 1) // 128 - start // 128 + 1 <= lib.tile_atoms(box)
            covered = start + size
        assert rows <= covered < rows + 32
