"""The order of the grouped GEMMs' tiles: every tile once, and tiles that run side by side share their operands."""
import subprocess

import pytest

PROGRAM = r"""
#include "tile_order.h"
#include <stdio.h>
#include <stdlib.h>
int main(int, char** a) {
  const int rows = atoi(a[1]), cols = atoi(a[2]);
  for (int i = 0; i < rows * cols; ++i) {
    int r, c;
    cb_tile_order(i, rows, cols, r, c);
    printf("%d %d\n", r, c);
  }
}
"""


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 11), (7, 5), (8, 8), (9, 11), (64, 16), (80, 56), (257, 8)])
def test_tiles_side_by_side_share_their_operands(rows, cols, tmp_path):
    from colossalai_b200.kernel.loader import CSRC

    src, exe = tmp_path / "order.cpp", tmp_path / "order"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(rows), str(cols)], check=True, capture_output=True, text=True).stdout
    tiles = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert sorted(tiles) == [(r, c) for r in range(rows) for c in range(cols)]
    for i in range(0, len(tiles), 74):                        # the CTA pairs of a round
        side = tiles[i:i + 74]
        # at most three bands of eight row tiles and a run of column blocks; one column block after the other asks for up to 75
        assert len({r for r, _ in side}) + len({c for _, c in side}) <= 40


def test_both_products_of_a_group_take_it():
    from colossalai_b200.kernel.loader import CSRC

    assert (CSRC / "grouped_gemm_tcgen05.cu").read_text().count("cb_tile_order(") == 2
