// Which kernel a forward's expert GEMMs take, from sizes the host knows: plain functions, so that the CPU test-suite
// checks the lines against the measurements beside them.
#pragma once
#include <stdint.h>

namespace atenia {

// INT8 calls of `rows` rows (tokens x experts per token) in a layer of `experts` experts: does the integer-MMA decode
// kernel (bf16_decode_gemm.cu) pay?  Up to 128 rows it always has.  Above, it passes an expert's weights through once per
// 32 rows of a group, so it needs experts large enough that widening them costs more than its own extra launches
// (digits, and a reduce pass where tiles are cut), and groups small enough for one or two passes.  One forward on a
// B200, integer-MMA / tensor-memory kernel, us:
//   d x F 4096 x 14336  8 experts, 130 / 192 / 256 rows 267 / 377, 284 / 379, 319 / 389; 4 experts, 160 / 224 271 / 280,
//                       219 / 284; 3 experts, 160 / 192 236 / 240, 267 / 243; 2 experts, 130 / 192 / 256 212 / 212, 228 / 220,
//                       277 / 227
//   2048 x 7168         8 experts, 130 / 192 / 250 118 / 156, 129 / 157, 140 / 159
//   2048 x 4096         8 experts, 130 / 192 / 250 90 / 102, 98 / 101, 106 / 103; 4 experts, 144 / 192 84 / 83, 88 / 84
//   2048 x 1408         64 experts, 132 / 192 177 / 180, 194 / 187; with a shared expert beside them 202 / 202, 222 / 224;
//                       60 experts and a shared one, 132 / 192 / 256 203 / 228, 220 / 244, 230 / 263; 32 experts, 192 / 252
//                       116 / 116, 120 / 118
//   smaller             1024 x 2816, 8 experts, 192 76 / 72; 1024 x 1024, 8 experts, 192 56 / 44; 2048 x 768, 128 experts,
//                       192 257 / 200; 512 x 1408, 8 experts, 192 62 / 43
// (The widening kernels split by rows per group as before: `rows` is all this rule and the row gather look at, so that
// every rank of a replicated batch and a single GPU choose alike.)
constexpr int kI8DecodeAlwaysRows = 128;
inline bool i8_decode_pays(int rows, int experts, int d, int F, bool shared) {
  if (rows <= kI8DecodeAlwaysRows) return true;
  const int64_t weights = (int64_t)d * F, r = rows, e = experts;
  if (weights >= (int64_t)1 << 25) return r < 64 * e;
  if (weights >= (int64_t)1 << 23) return r <= 30 * e;
  return shared && weights >= (int64_t)1 << 21 && r <= 5 * e;
}

}  // namespace atenia
