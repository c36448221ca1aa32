// Four values to four int8 codes, packed: code = clamp(round_half_away(x / s), -127, 127) with inv ~ 1 / s,
// without a division (or a multi-instruction roundf) per value.
//
// x * inv is within 2^-22 relative of the quotient the reference rounds (two roundings of half an ulp each),
// i.e. within 4e-5 for |x / s| <= 128, so the nearest integer of the product IS the code unless the product
// lies closer than that to a half-integer.  The nearest integer comes from one fused multiply-add with
// 1.5 * 2^23 (the sum's low byte is the code in two's complement), the distance to it from two more operations;
// values more than 0.4999 away, and NaNs, take `exact`, the reference's own sequence: 2 values in 10 000.
#pragma once
#include <stdint.h>

namespace atenia {

template <typename Exact>
__device__ __forceinline__ uint32_t round_codes4(const float (&x)[4], const float (&inv)[4], Exact exact) {
  constexpr float kMagic = 12582912.0f;
  uint32_t b[4];
  bool sure = true;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float y = __fmaf_rn(x[j], inv[j], kMagic);
    const float off = __fmaf_rn(x[j], inv[j], -__fsub_rn(y, kMagic));
    sure = sure && fabsf(off) <= 0.4999f;
    b[j] = __float_as_uint(y);
  }
  if (!sure) {
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = (uint32_t)exact(x[j], j);
  }
  return __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}

}  // namespace atenia
