// Digits of the integer router (router_i8.cu): the grids, which values lie on them, and the way back.  Written once for the
// device and for the CPU test-suite, which compiles this header by itself.
//
//   x[t, k] = 2^(ex - 30) X,  |X| < 2^30, four balanced base-256 digits; ex from the largest bf16 value of the token's k-range
//   w[e, k] = 2^(ew - 38) W,  |W| <= 2^38, five digits; ew from the largest f32 value of the row
// A value is on its grid when X (W) is an integer: every bf16 value from 2^(ex - 23) up, every f32 value from 2^(ew - 15) up,
// smaller ones where enough of their low bits are zero.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define ATENIA_HD __host__ __device__
#else
#define ATENIA_HD
#endif

namespace atenia {

// ex of a k-range from the bits (without the sign) of its largest value; k-ranges below 2^-89 keep that grid
ATENIA_HD inline int digits_x_exponent(uint32_t largest) {
  const int field = (int)(largest >> 7);
  return (field < 37 ? 37 : field) - 126;
}
// Bits (without the sign) from which on a value is on the grid for sure
ATENIA_HD inline uint32_t digits_x_edge(int ex) { return 104 + ex > 0 ? (uint32_t)(104 + ex) << 7 : 0u; }
// Can a value with these bits be off the grid?  `smallest`: the smallest of the k-range but zeros; 0: none.
ATENIA_HD inline bool digits_x_off_grid(uint32_t smallest, int ex) { return smallest != 0 && smallest < digits_x_edge(ex); }
// Two bf16 values (without the signs) as keys whose minimum, as signed halves, is the smallest value but zeros (a zero has the
// largest key)
ATENIA_HD inline uint32_t digits_keys(uint32_t two) { return two + 0x7fff7fffu; }
ATENIA_HD inline uint32_t digits_of_key(uint32_t key) { return (key - 0x7fffu) & 0xffffu; }

// The bytes of the result are the balanced digits of X, top digit in the top byte.
ATENIA_HD inline uint32_t digits_x_bytes(int32_t X) { return ((uint32_t)X + 0x80808080u) ^ 0x80808080u; }
// The lowest balanced digit, in [-128, 127], taken off W
ATENIA_HD inline int8_t digits_w_next(long long& W) {
  const long long dg = ((W + 128) & 255) - 128;
  W = (W - dg) >> 8;
  return (int8_t)dg;
}
// Sums A_s of the digit products of level s (plane i of x and j of w: s = i + j): X . W = 2^40 (p[0] + 2^-24 p[1] + 2^-40 p[2]),
// each p below 2^51 in magnitude
ATENIA_HD inline void digits_fold(const int32_t (&A)[8], long long (&p)[3]) {
  p[0] = (long long)A[0] * 65536 + (long long)A[1] * 256 + A[2];
  p[1] = (long long)A[3] * 65536 + (long long)A[4] * 256 + A[5];
  p[2] = (long long)A[6] * 256 + A[7];
}

}  // namespace atenia
