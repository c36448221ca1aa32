// Token tiles of the CTA-pair kernel (grouped_gemm_2cta.cu) and the TMA boxes that load them, written once for the
// device, for the host that encodes the boxes and for the CPU test-suite, which compiles this header by itself.
#pragma once

#if defined(__CUDACC__)
#define ATENIA_HD __host__ __device__
#else
#define ATENIA_HD
#endif

namespace atenia {

constexpr int kPairTokens = 256;  // token rows of a tile at most (MMA N)
// The token rows are described by boxes of several heights; a tile takes the smallest that holds half of it.
constexpr int kPairBoxes = 8;
ATENIA_HD constexpr int pair_box_rows(int box) { return 16 * (box + 1); }

// A group of `rows` rows is cut into equal tiles of a multiple of 16 rows, so none is a nearly empty remainder.  `most`:
// the token rows a stage of the launch's ring has room for (pair_tokens).
ATENIA_HD inline int pair_tiles(int rows, int most = kPairTokens) { return (rows + most - 1) / most; }
ATENIA_HD inline int pair_tile_rows(int rows, int tiles) { return tiles > 0 ? ((rows + tiles - 1) / tiles + 15) & ~15 : 16; }
// MMA N of a tile of `rows` rows, and the box that holds the half of it which one CTA of the pair stages
ATENIA_HD inline int pair_tile_n(int rows) { return (rows + 15) & ~15; }
ATENIA_HD inline int pair_tile_box(int n) { return (n / 2 + 15) / 16 - 1; }

// Boxes (bit i: box i) that the tiles of one group of `rows` rows use: that of the full tiles and that of the last.
inline unsigned pair_boxes_of_group(int rows, int most = kPairTokens) {
  const int tiles = pair_tiles(rows, most);
  if (tiles < 1) return 0u;
  const int full = pair_tile_rows(rows, tiles), last = rows - (tiles - 1) * full;
  const unsigned of_last = 1u << pair_tile_box(pair_tile_n(last));
  return tiles > 1 ? of_last | 1u << pair_tile_box(pair_tile_n(full)) : of_last;
}
constexpr unsigned kPairAllBoxes = (1u << kPairBoxes) - 1u;  // rows known on the device only

}  // namespace atenia
