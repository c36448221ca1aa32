// Fragments of the f64 tensor-core routers (router_dmma.cu, router_splitk.cu).
#pragma once
#include <type_traits>

#include "common.cuh"

namespace atenia {

template <int I>
using Int = std::integral_constant<int, I>;

// D[8x8] += A[8x4] * B[4x8].  Lane l holds A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// N consecutive 32-bit words (N = 4 or 8) from a 16-byte aligned address
template <int N, bool LDG>
__device__ __forceinline__ void ld_words(uint32_t (&w)[N], const void* p) {
#pragma unroll
  for (int i = 0; i < N / 4; ++i) {
    const uint4 v = LDG ? __ldg(static_cast<const uint4*>(p) + i) : static_cast<const uint4*>(p)[i];
    w[4 * i] = v.x;
    w[4 * i + 1] = v.y;
    w[4 * i + 2] = v.z;
    w[4 * i + 3] = v.w;
  }
}
template <int N>
__device__ __forceinline__ void zero_words(uint32_t (&w)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) w[i] = 0u;
}
// element j (a constant after unrolling) of a lane's eight consecutive x values held as raw words
template <bool XF, int N>
__device__ __forceinline__ double x_elem(const uint32_t (&w)[N], int j) {
  if (XF) return (double)__uint_as_float(w[j]);
  return (double)((j & 1) ? bf16hi(w[j >> 1]) : bf16lo(w[j >> 1]));
}

}  // namespace atenia
