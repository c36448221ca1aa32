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
// How a launch deals its tiles to the pairs when one more group, whose tiles may be longer, comes with it: round by round, the
// extra group's first; the pairs that have one in the last of their rounds miss as many rounds as it lasts (`weight`).
struct PairDeal {
  int pairs, full, rest, weight;  // pairs of SMs; rounds of extra tiles, and those of one more round
};
ATENIA_HD inline PairDeal pair_deal(int pairs, int extra_tiles, int extra_k_blocks, int k_blocks) {
  const int full = extra_tiles / pairs, weight = (extra_k_blocks + k_blocks / 2) / k_blocks;
  return PairDeal{pairs, full, extra_tiles - full * pairs, weight < 1 ? 1 : weight};
}
// The `i`-th tile of `pair`: of the extra group (`extra`), or of the others, counted from 0 each.
ATENIA_HD inline int pair_deal_tile(const PairDeal& d, int pair, int i, bool& extra) {
  const int m = i - d.full;  // rounds after the full ones
  extra = m < 0 || (m == 0 && pair < d.rest);
  if (extra) return pair + i * d.pairs;
  const int others = d.pairs - d.rest, late = d.weight * others;
  return pair < d.rest ? late + (m - 1) * d.pairs + pair
         : m < d.weight ? m * others + pair - d.rest : late + (m - d.weight) * d.pairs + pair;
}

constexpr unsigned kPairAllBoxes = (1u << kPairBoxes) - 1u;  // rows known on the device only

}  // namespace atenia
