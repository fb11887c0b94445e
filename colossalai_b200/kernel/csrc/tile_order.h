// The order in which the tiles of one product are taken: bands of CB_BAND row tiles, in a band the row tiles of one column block after
// the other.  CTAs that run at the same time then share their operands: 74 tiles side by side ask for some 18 blocks of rows and
// columns, where all row tiles of a column block in turn are up to 75 of them - every round of CTAs all rows once more, which is
// memory traffic once the rows do not fit in L2.  Plain C++ beside CUDA, so that the order can be looked at on the host.
#pragma once

#ifdef __CUDACC__
#define CB_TILE_ORDER __host__ __device__ __forceinline__
#else
#define CB_TILE_ORDER inline
#endif

constexpr int CB_BAND = 8;

CB_TILE_ORDER void cb_tile_order(int local, int row_tiles, int col_blocks, int& row_tile, int& col_block) {
  int first = 0, rows = row_tiles;
  if (row_tiles > CB_BAND) {                 // (a group of one band, as most are, is spared the division)
    const int band = local / (CB_BAND * col_blocks);
    first = band * CB_BAND;
    local -= first * col_blocks;
    rows = row_tiles - first < CB_BAND ? row_tiles - first : CB_BAND;
  }
  col_block = local / rows;
  row_tile = first + local - col_block * rows;
}
