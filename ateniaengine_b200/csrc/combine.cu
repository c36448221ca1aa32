// Combine: gate-weighted sum of a token's expert outputs back in token order, plus the shared expert.
//
// The reference accumulates out[d] += w * y_e[d] over the selected experts in ascending expert order
// with an f32 multiply followed by an f32 add (src/moe/sparse.rs:227-233), then adds scale * shared
// (src/moe/layer.rs:415-429).  The kernel gathers each token's k rows from the dispatch-ordered
// buffer in slot order (slots are ascending experts) and repeats that arithmetic, so the result does
// not depend on scheduling: no atomics.
//
// Also here: the small elementwise kernels of the library (int8 per-row quantiser, f32 to bf16 conversion).
#include "common.cuh"
#include "round_codes.cuh"

namespace atenia {
namespace {

// One block per token, one 16-byte vector of the row per thread and step.  K is the top-k count (a
// compile-time bound so that the k row loads of a vector are all issued before the first is used);
// the arithmetic order does not depend on it.
template <int K>
__global__ void __launch_bounds__(256) combine_kernel(CombineArgs a) {
  const int t = blockIdx.x;
  const int nvec = a.d / 8;
  chain_next();
  chain_wait();
  int rows[K];
  float w[K];
#pragma unroll
  for (int s = 0; s < K; ++s) {
    rows[s] = s < a.k ? a.inv_perm[(size_t)t * a.k + s] : -1;
    w[s] = s < a.k ? a.topk_w[(size_t)t * a.k + s] : 0.f;
  }
  const float scale = a.gate_scale ? a.gate_scale[t] : 1.0f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    uint4 y[K];
#pragma unroll
    for (int s = 0; s < K; ++s)
      if (rows[s] >= 0) y[s] = *reinterpret_cast<const uint4*>(a.y_rows + (size_t)rows[s] * a.d + v * 8);
    uint4 ysh = make_uint4(0, 0, 0, 0);
    if (a.y_shared) ysh = *reinterpret_cast<const uint4*>(a.y_shared + (size_t)t * a.d + v * 8);
    float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
    if (a.residual) {
      const float4* r = reinterpret_cast<const float4*>(a.residual + (size_t)t * a.d + v * 8);
      r0 = r[0];
      r1 = r[1];
    }
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
    for (int s = 0; s < K; ++s) {
      if (rows[s] < 0) continue;  // slot past k, or an entry without a row (invalid expert id, reported by the dispatch)
      const uint32_t p[4] = {y[s].x, y[s].y, y[s].z, y[s].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * j] = __fadd_rn(acc[2 * j], __fmul_rn(w[s], bf16lo(p[j])));
        acc[2 * j + 1] = __fadd_rn(acc[2 * j + 1], __fmul_rn(w[s], bf16hi(p[j])));
      }
    }
    if (a.y_shared) {
      const uint32_t p[4] = {ysh.x, ysh.y, ysh.z, ysh.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * j] = __fadd_rn(acc[2 * j], __fmul_rn(scale, bf16lo(p[j])));
        acc[2 * j + 1] = __fadd_rn(acc[2 * j + 1], __fmul_rn(scale, bf16hi(p[j])));
      }
    }
    if (a.residual) {
      acc[0] = __fadd_rn(acc[0], r0.x); acc[1] = __fadd_rn(acc[1], r0.y);
      acc[2] = __fadd_rn(acc[2], r0.z); acc[3] = __fadd_rn(acc[3], r0.w);
      acc[4] = __fadd_rn(acc[4], r1.x); acc[5] = __fadd_rn(acc[5], r1.y);
      acc[6] = __fadd_rn(acc[6], r1.z); acc[7] = __fadd_rn(acc[7], r1.w);
    }
    if (a.out_is_f32) {
      float4* o = reinterpret_cast<float4*>(static_cast<float*>(a.out) + (size_t)t * a.d + v * 8);
      o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
      uint4* o = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.out) + (size_t)t * a.d + v * 8);
      *o = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                      pack_bf16x2(acc[6], acc[7]));
    }
  }
}

// One block per row: scale = max|row| / 127 (1 for a zero row), q = clamp(round_half_away(w * (1/scale))).
// The row is read once: a thread keeps its (up to kQuantVecs) groups of four values in registers between the
// maximum and the rounding; what a longer row has beyond that is read again.  HBM-bound, 5 bytes per weight.
// VEC: every row starts on a 16-byte boundary (a thread's four values are one vector), else single values, a
// block width apart.  Narrow rows take narrower blocks, so that several rows share an SM.  Measured on a B200:
// 14336 x 4096 93 -> 50 us (floor 47), against a kernel that read every row twice with 4-byte loads.
constexpr int kQuantVecs = 8;

template <bool VEC>
__global__ void __launch_bounds__(512) quantize_rows_kernel(const float* __restrict__ w, int64_t cols,
                                                            int8_t* __restrict__ q, float* __restrict__ scales) {
  __shared__ float red[16];
  const int64_t r = blockIdx.x;
  const float* row = w + r * cols;
  int8_t* qrow = q + r * cols;
  // value j of a thread's vector v
  auto col_of = [&](int v, int j) -> int64_t {
    const int64_t base = (int64_t)v * blockDim.x * 4;
    return VEC ? base + threadIdx.x * 4 + j : base + threadIdx.x + (int64_t)j * blockDim.x;
  };
  auto load = [&](int v) -> float4 {
    if (VEC) return col_of(v, 0) < cols ? *reinterpret_cast<const float4*>(row + col_of(v, 0)) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(col_of(v, 0) < cols ? row[col_of(v, 0)] : 0.f, col_of(v, 1) < cols ? row[col_of(v, 1)] : 0.f,
                       col_of(v, 2) < cols ? row[col_of(v, 2)] : 0.f, col_of(v, 3) < cols ? row[col_of(v, 3)] : 0.f);
  };
  auto amax4 = [](float m, const float4& x) {
    return fmaxf(fmaxf(m, fmaxf(fabsf(x.x), fabsf(x.y))), fmaxf(fabsf(x.z), fabsf(x.w)));
  };
  const int nvec = (int)((cols + (int64_t)blockDim.x * 4 - 1) / ((int64_t)blockDim.x * 4));
  float4 keep[kQuantVecs];
  float amax = 0.f;
#pragma unroll
  for (int v = 0; v < kQuantVecs; ++v) keep[v] = v < nvec ? load(v) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int v = 0; v < kQuantVecs; ++v) amax = amax4(amax, keep[v]);
  for (int v = kQuantVecs; v < nvec; ++v) amax = amax4(amax, load(v));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  float m = red[0];
  for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = fmaxf(m, red[i]);
  const float scale = m > 0.f ? __fdiv_rn(m, 127.0f) : 1.0f;
  if (threadIdx.x == 0) scales[r] = scale;
  const float inv = __fdiv_rn(1.0f, scale);
  const float inv4[4] = {inv, inv, inv, inv};
  auto exact = [&](float x, int) -> int {
    float v = roundf(__fmul_rn(x, inv));  // roundf: halves away from zero, like Rust's f32::round
    v = fminf(fmaxf(v, -127.0f), 127.0f);
    return (int)v;
  };
  auto store = [&](int v, const float4& x) {
    const float x4[4] = {x.x, x.y, x.z, x.w};
    const uint32_t p = round_codes4(x4, inv4, exact);
    if (VEC) {
      if (col_of(v, 0) < cols) *reinterpret_cast<uint32_t*>(qrow + col_of(v, 0)) = p;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col_of(v, j) < cols) qrow[col_of(v, j)] = (int8_t)(p >> (8 * j));
    }
  };
#pragma unroll
  for (int v = 0; v < kQuantVecs; ++v)
    if (v < nvec) store(v, keep[v]);
  for (int v = kQuantVecs; v < nvec; ++v) store(v, load(v));
}

// Eight values per thread and step where both sides are on a 16-byte boundary, single values for the rest.
__global__ void f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
  const int64_t n8 = vec ? n / 8 : 0;
  for (int64_t i = first; i < n8; i += stride) {
    const float4 a = reinterpret_cast<const float4*>(src)[2 * i], b = reinterpret_cast<const float4*>(src)[2 * i + 1];
    reinterpret_cast<uint4*>(dst)[i] =
        make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  }
  for (int64_t i = 8 * n8 + first; i < n; i += stride) dst[i] = __float2bfloat16(src[i]);
}

}  // namespace

int launch_combine(const CombineArgs& a, cudaStream_t s) {
  if (a.T <= 0) return ATENIA_OK;
  // d / 8 vectors per token: narrow rows take narrower blocks
  const int nvec = a.d / 8;
  const int threads = nvec >= 256 ? 256 : nvec >= 128 ? 128 : 64;
  auto launch = [&](auto kernel) { return launch_chained(a.chained, kernel, dim3(a.T), dim3(threads), 0, s, a); };
  int rc;
  if (a.k <= 2) rc = launch(combine_kernel<2>);
  else if (a.k <= 4) rc = launch(combine_kernel<4>);
  else if (a.k <= 6) rc = launch(combine_kernel<6>);
  else rc = launch(combine_kernel<8>);
  count_launch();
  return rc;
}

__global__ void set_pair_kernel(int32_t* p, int32_t a, int32_t b) {
  p[0] = a;
  p[1] = b;
}

int launch_set_pair(int32_t* p, int32_t a, int32_t b, cudaStream_t s) {
  set_pair_kernel<<<1, 1, 0, s>>>(p, a, b);
  count_launch();
  return (int)cudaGetLastError();
}

int launch_f32_to_bf16(const float* src, __nv_bfloat16* dst, int64_t n, cudaStream_t s) {
  if (n <= 0) return ATENIA_OK;
  const int64_t want = (n + 2047) / 2048;  // blocks of eight values a thread
  const int blocks = (int)(want < 148 * 8 ? want : 148 * 8);
  f32_to_bf16_kernel<<<blocks, 256, 0, s>>>(src, dst, n);
  count_launch();
  return (int)cudaGetLastError();
}

}  // namespace atenia

extern "C" int atenia_quantize_per_row_i8(const float* w, int64_t rows, int64_t cols, int8_t* q, float* scales,
                                          void* stream) {
  if (!w || !q || !scales) return ATENIA_ERR_NULL;
  if (rows < 0 || cols <= 0 || rows > 0x7fffffff) return ATENIA_ERR_SHAPE;
  if (rows == 0) return ATENIA_OK;
  // the narrowest block whose registers hold a row (32 values per thread)
  const int threads = cols <= 64 * 32 ? 64 : cols <= 128 * 32 ? 128 : cols <= 256 * 32 ? 256 : 512;
  const bool vec = cols % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0 && (reinterpret_cast<uintptr_t>(q) & 3u) == 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (vec) atenia::quantize_rows_kernel<true><<<(unsigned)rows, threads, 0, s>>>(w, cols, q, scales);
  else atenia::quantize_rows_kernel<false><<<(unsigned)rows, threads, 0, s>>>(w, cols, q, scales);
  atenia::count_launch();
  return (int)cudaGetLastError();
}
