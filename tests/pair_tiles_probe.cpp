// Test-only: compiles the tile arithmetic of the CTA-pair kernel with a host compiler.  Not part of the product library.
#include "../ateniaengine_b200/csrc/pair_tiles.cuh"

extern "C" unsigned pair_probe_mask(int rows) { return atenia::pair_boxes_of_group(rows); }
// The kernel's walk over the tiles of a group: row0, rows and box of each; returns the number of tiles.
extern "C" int pair_probe_walk(int rows, int* row0, int* n_rows, int* box, int* half) {
  const int tiles = atenia::pair_tiles(rows), height = atenia::pair_tile_rows(rows, tiles);
  for (int i = 0; i < tiles; ++i) {
    row0[i] = i * height;
    n_rows[i] = rows - row0[i] < height ? rows - row0[i] : height;
    const int n = atenia::pair_tile_n(n_rows[i]);
    half[i] = n / 2;
    box[i] = atenia::pair_tile_box(n);
  }
  return tiles;
}
// The kernel's deal of tiles beside an extra group: the i-th tile of a pair; returns 1 where it is the extra group's.
extern "C" int pair_probe_deal(int pairs, int extra_tiles, int extra_kb, int kb, int pair, int i, int* tile) {
  bool extra;
  *tile = atenia::pair_deal_tile(atenia::pair_deal(pairs, extra_tiles, extra_kb, kb), pair, i, extra);
  return extra;
}
