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

// bf16 products above decode size: the CTA-pair kernel (grouped_gemm_2cta.cu) against the single-CTA one
// (grouped_gemm.cu).  The pair kernel's tile is 256 weight rows x up to 256 tokens and leaves tensor memory two bytes a
// lane; over a short k that store takes longer than the MMAs.  One product on a B200, pair / single-CTA, us:
//   k 512   8 experts, n 1408, 32 / 64 / 256 rows an expert 16 / 14, 17 / 14, 27 / 20; n 512, 64 rows 13 / 14; 128 experts, n 512,
//           16 / 100 / 512 rows 49 / 43, 64 / 46, 143 / 97
//   k 1024  8 experts, n 1024, 64 / 128 / 256 rows 16 / 18, 18 / 18, 27 / 25; 32 experts, n 2816, 64 / 256 / 1024 rows 74 / 72, 128 /
//           120, 388 / 344; 128 experts, n 512, 100 / 256 rows 77 / 68, 109 / 97
//   k 1408  (n 2048) 32 experts, 64 / 256 rows 45 / 43, 69 / 73; 128 experts, 100 / 256 157 / 142, 216 / 255
//   k 2048  8 experts, n 512, 64 rows 18 / 22; 32 experts, n 1408, 64 / 256 / 1024 rows 74 / 78, 109 / 117, 293 / 345
// Groups of 512 rows or more take the pair kernel with the rows as its M side (grouped_gemm_pair_rows.cu).
// A shared expert's gate/up product (`beside` the routing kernels, on the second stream) keeps the transposed pairs up to 4096
// tokens; a forward with it there / on the single-CTA kernel, us: 32 experts top-4 of 1024 x 1024, shared 4096, 1184 / 2048 / 3000 /
// 4096 tokens 119 / 134, 163 / 173, 215 / 222, 268 / 261; of 512 x 1408, shared 2816, 1024 / 3000 86 / 100, 140 / 146; 16 experts
// top-1 of 1024 x 2048, shared 2048, 1500 / 4096 96 / 102, 147 / 159.
enum Bf16Kernel { kBf16Pairs = 0, kBf16Single = 1, kBf16PairRows = 2 };
inline Bf16Kernel bf16_product_kernel(int rows, int groups, int k, bool beside) {
  if (k > 1024 || rows < (beside ? 4096 : 1024)) return kBf16Pairs;
  return (int64_t)rows >= (int64_t)512 * groups ? kBf16PairRows : kBf16Single;
}

// Token rows of the CTA-pair kernel's tiles at most, and with them the depth of its ring: 256 (6 stages), 192 (7), 128 (8) or 64 (10).
// With few rows per group the kernel streams weights, and what limits that is the bytes in flight (a stage holds 16 KiB of
// weights per SM and 128, 64 or 32 token rows); a group of more rows than the tile passes its weights through twice.
// One forward on a B200, 256 / 128 / 64, us (rows a group):
//   8 experts of 4096 x 14336   16 tokens (4) 451 / 432 / 422, 120 (30) 464 / 444 / 436, 180 (45) 476 / 456 / 455, 256 (64)
//                               488 / 466 / 535, 350 (87) 519 / 503 / 584, 400 (100) 530 / 548 / 602
//   60 of 2048 x 1408, shared   16 (1) 147 / 138 / 137, 150 (10) 209 / 197 / 195, 220 (15) 217 / 201 / 203, 333 (22) 237 / 223 / 228,
//                               1300 (87) 309 / 297 / 380, 1500 (100) 315 / 296 / 370, 1700 (113) 351 / 356 / 423
//   64 of 2048 x 1408, shared   61 (6) 205 / 196 / 196, 300 (28) 227 / 218 / 218, 900 (84) 272 / 269 / 317, 1300 (122) 306 / 310 / 380
// ... and 256 / 192 / 128: 8 experts of 4096 x 14336, 350 tokens (87) 501 / 493 / 490, 400 (100) 512 / 502 / 543, 500 (125)
// 594 / 549 / 606, 600 (150) 618 / 674 / 651; 60 of 2048 x 1408, 1300 (87) 297 / 292 / 292, 1700 (113) 341 / 334 / 337, 2048
// (137) 372 / 372 / 410, 2500 (167) 429 / 442 / 491; 64, 1300 (122) 305 / 302 / 305, 1700 (159) 343 / 335 / 380, 2000 (187) 389
// / 415 / 435.
// A product whose tiles all run at once takes the lowest that still do (8 experts of 512 x 1408, 600 / 1000 tokens 38.3 / 35.2 /
// 35.2, 42.6 / 37.7 / 37.5).  Also beside others: a shared expert of 2816 on the second stream of 32 experts of 512 x 1408, 333 tokens
// over 22 feature tiles (64-row tiles would take two rounds) 66.1 / 66.8 / 68.0; with both its products in 256-row tiles 500 / 700 /
// 1480 tokens 73.4 -> 77.4, 82.5 -> 88.9, 105.1 -> 109.1.
constexpr int64_t kPairs = 74;
inline int pair_tokens_of(int rows, int groups, int f_tiles) {
  for (int t = 64; t <= 128; t += 64)
    if (f_tiles * (int64_t)(groups == 1 ? (rows + t - 1) / t : groups + rows / t) <= kPairs) return t;
  if (groups == 1) return rows <= 64 ? 64 : rows <= 128 ? 128 : 256;
  const int64_t r = rows, g = groups;
  if (r <= 12 * g || (g <= 16 && r <= 36 * g)) return 64;
  return r <= 88 * g ? 128 : r <= 140 * g ? 192 : 256;
}

// Does the shared expert's group, cut by the routed groups' tile height, ride along in their launches (merges_shared)?  It
// passes its weights through once per tile of its rows, its own launches on the second stream once per 256: the passes more are
// traffic that its missing launches (some 8 us) and the interleaving have to pay for.  B200, a forward along / aside, us, by what
// those passes read in MB:
//   64-row tiles   64 top-1 experts of 2048 x 1408, shared 1408, 600 tokens (120) 209 / 222; shared 5632, 100 (70) 152 / 157, 300 (210)
//                  205 / 203, 600 (480) 237 / 230; shared 22528, 100 (280) 206 / 202, 300 (830) 276 / 261, 600 (1940) 405 / 329; 128 top-1
//                  of 2048 x 768, shared 768, 600 (66) 236 / 251; shared 3072, 1000 (450) 273 / 261; shared 12288, 100 (150) 160 / 165,
//                  300 (450) 245 / 241, 600 (1060) 325 / 287; 16 top-1 of 1024 x 2816, shared 5632, 303 (100) 85 / 87, 500 (210) 87 / 93; 32
//                  top-2 of 2048 x 1408, shared 11264, 100 (140) 136 / 145
//   higher ones    64 top-1 of 2048 x 1408, shared 5632, 1000 (280) 257 / 263; shared 22528, 1000 (1110) 423 / 405, 1480 (1660) 572 / 530; 64
//                  top-2, shared 22528, 1000 (1110) 424 / 412, 1480 (1660) 591 / 548; 16 top-1 of 2048 x 4096, shared 8192, 600 (200) 199 /
//                  215, 1000 (400) 242 / 249; 32 top-2 of 2048 x 1408, shared 11264, 600 (280) 181 / 193
inline bool shared_rides_along(int tokens, int tile, int d, int Fs) {
  const int64_t more = (tokens + tile - 1) / tile - (tokens + 255) / 256;
  return more * 6 * d * Fs <= (int64_t)(tile == 64 ? 240 : 576) * 1000000;
}

// Does the integer router (router_i8.cu) pay?  It computes 64 rows whatever E is, and has a floor of some 15 us; the f64 routers' time
// follows T, d and E.  B200, router kernel, it / the f64 one of that size, us (forwards where the kernels are close):
//   33 - 64 experts, 1185 - 2368 tokens   (64) d 2048, 1185 / 1600 / 2048 tokens 21.1 / 27.0, 21.0 / 30.5, 28.0 / 30.8; 1536, 1185 / 1600 /
//            2368 20.5 / 21.3, 20.9 / 24.5, 25.3 / 25.0; 1024, 1300 / 2048 17.2 / 17.8, 21.8 / 19.4; 768, 1600 16.9 / 14.2; 256, 2048 16.7 / 8.9
//   ... more tokens   d 2048, 4096 / 8192 30.3 / 54, 46.6 / 104; 1536, 2400 25.3 / 42.1; 768, 2400 21.1 / 24.9; 512, 3000 / 4096 forwards
//            equal, 8192 128 / 138; 256, 4096 / 8192 forwards 80 / 76, 107 / 109
//   17 - 32 experts, more than 2368   (32) d 4096, 3000 / 4096 40.5 / 51.4, 43.6 / 51.6; 2048, 2400 / 8192 26.0 / 28.0, 45.4 / 54.7;
//            1536, 4096 / 8192 24.5 / 23.2, 38.3 / 43.8; 1024, 4096 / 8192 forwards 68 / 66, 102.5 / 104.3; 512, 8192 78 / 76
inline bool router_i8_pays(int tokens, int d, int experts) {
  const int64_t work = (int64_t)tokens * d;
  if (tokens <= 8 * 148 || experts <= 16) return false;
  if (tokens <= 16 * 148) return experts > 32 && d >= 1536;
  return experts > 32 ? d >= 768 || work >= 1 << 21 : d >= 2048 || work >= 1 << 23;
}

}  // namespace atenia
