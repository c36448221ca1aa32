// Dense W8A16 weight quantiser and its materialising dequant: the [K, N] row-major layout with one
// scale per (group of consecutive rows, column) that the reference uses for non-MoE linear weights
// (src/tensor/quantizer.rs:67-118 per channel, :176-246 per group; src/cuda/int8_to_bf16.cu:24-40,
// :99-117).  The MoE tiers use the per-row layout of combine.cu instead.
//
// Both directions are streaming, HBM-bound work (algorithmic bytes per weight: quantise 4 + 1, dequant 1 + 2):
//   quantize_groups  a block owns 32 to 128 columns x one group; the group's values stay in registers between the
//                    maximum and the rounding, so the matrix is read once (groups of at most 128 rows)
//   quantize_tall    a cluster of one to eight blocks owns 64 columns x one taller group and reads it twice, the
//                    second time from L2 where it fits
//   quantize_passes  maxima, scales and codes in three launches over the whole grid, for matrices whose groups
//                    and strips are too few for the kernel above
//   dequant          a block owns 256 columns x 64 rows; a lane keeps its eight scales while the group lasts;
//                    narrow matrices and groups of few rows take a flat walk
// The three passes and the flat walk spend two 64-bit divisions per vector, the others none.  Measured on a B200
// at 4096 x 14336, groups of 128: quantise 149 (three passes) -> 51 us, dequant 42 (flat) -> 32 us; floors at the
// measured copy rate 47 and 28 us.
//   scale = max(amax / 127, 1e-12); q = clamp(round_half_away(w / scale), -127, 127), NaN -> 0;
//   bf16 = high half of (float)q * scale (truncation, as the reference's kernel does)
#include <cooperative_groups.h>

#include "common.cuh"
#include "round_codes.cuh"

namespace atenia {
namespace {

constexpr int COLS_PER_BLOCK = 128;  // three passes: 32 lanes x 4 columns
constexpr int GROUP_ROWS_MAX = 128;  // tallest group that stays in registers: 16 row lanes x 8 rows
constexpr int TALL_WARPS = 16;
constexpr int TALL_COLS = 64;        // 16 lanes x 4 columns: a warp covers two rows
constexpr int DEQ_COLS = 256, DEQ_ROWS = 64;

// Four columns of a row per lane (LANES lanes side by side): consecutive ones as one vector (VEC: every row
// starts on a 16-byte boundary), else LANES apart.  Columns >= N read as 0.
template <bool VEC, int LANES>
__device__ __forceinline__ int64_t col_of(int64_t strip0, int lane, int j) {
  return VEC ? strip0 + lane * 4 + j : strip0 + lane + LANES * j;
}
template <bool VEC, int LANES>
__device__ __forceinline__ void load_cols4(float (&v)[4], const float* __restrict__ row, int64_t strip0, int lane,
                                           int64_t N) {
  if (VEC) {
    const int64_t c = strip0 + lane * 4;
    const float4 f = c < N ? *reinterpret_cast<const float4*>(row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t c = strip0 + lane + LANES * j;
      v[j] = c < N ? row[c] : 0.f;
    }
  }
}

__device__ __forceinline__ int quantize_one(float w, float s) {
  float v = roundf(__fdiv_rn(w, s));  // roundf: halves away from zero, like Rust's f32::round
  if (v != v) return 0;               // Rust's `as i32` sends NaN to 0
  v = fminf(fmaxf(v, -127.0f), 127.0f);
  return (int)v;
}

template <bool VEC, int LANES>
__device__ __forceinline__ void store_codes4(const float (&w)[4], const float* s, const float (&inv)[4],
                                             int8_t* __restrict__ row, int64_t strip0, int lane, int64_t N) {
  const uint32_t p = round_codes4(w, inv, [&](float x, int j) { return quantize_one(x, s[j]); });
  if (VEC) {
    const int64_t c = strip0 + lane * 4;
    if (c < N) *reinterpret_cast<uint32_t*>(row + c) = p;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t c = strip0 + lane + LANES * j;
      if (c < N) row[c] = (int8_t)(p >> (8 * j));
    }
  }
}

// A NaN is skipped, as in the reference: fmaxf returns the other operand, and nothing compares greater for one.  The groups kernel is
// faster with the first form, the tall one with the second (4096 x 14336 by 128 / 64 51.4 / 52.0, 49.9 / 51.9 us; 8192 x 14336 by
// 512 / 1024 / 4096 143.5 / 140.7, 150.2 / 147.2, 167.2 / 163.6).
template <bool COMPARE>
__device__ __forceinline__ void max_cols4(float (&m)[4], const float (&v)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a = fabsf(v[j]);
    if (!COMPARE) m[j] = fmaxf(m[j], a);
    else if (a > m[j]) m[j] = a;
  }
}
__device__ __forceinline__ float scale_of(float amax) { return fmaxf(__fdiv_rn(amax, 127.0f), 1e-12f); }

// A block of LANES x RL threads owns 4 LANES columns x one group of at most RL * GROUP_RPT rows.  HBM-bound as long as other
// blocks of the SM load while one rounds and stores, so blocks are small (many per SM, each at another point) and the
// rounding is kept short: one thread per column turns the RL partial maxima into the scale and its reciprocal, not every
// thread for its own four.  B200, 4096 x 14336 f32 (floor 45 us at the measured copy rate), blocks of 512 threads x 128
// columns with the scales in every thread / these: groups of 128 67.4 / 51.2 us, 100 75.7 / 55.6, 64 55.6 / 49.5, 48
// 63.8 / 55.6, 32 63.9 / 49.4, 20 84.9 / 59.3.  Sixteen rows per thread lose (128: 61), blocks twice as wide too (128: 53.4).
constexpr int GROUP_RPT = 8;
template <bool VEC, int LANES, int RL>
__global__ void __launch_bounds__(LANES * RL) quantize_groups_kernel(const float* __restrict__ w, int64_t K, int64_t N,
                                                                     int G, unsigned strips, int8_t* __restrict__ q,
                                                                     float* __restrict__ scales) {
  constexpr int COLS = LANES * 4;
  __shared__ __align__(16) float red[RL][COLS];
  __shared__ float4 scale_s[LANES], inv_s[LANES];
  const int lane = threadIdx.x % LANES, rl = threadIdx.x / LANES;
  const unsigned g = blockIdx.x / strips;
  const int64_t strip0 = (int64_t)(blockIdx.x - g * strips) * COLS;
  const int64_t lo = (int64_t)g * G;
  const int rows = (int)(K - lo < G ? K - lo : G);
  float v[GROUP_RPT][4];
#pragma unroll
  for (int i = 0; i < GROUP_RPT; ++i) {
    const int r = rl + RL * i;
    if (r < rows) load_cols4<VEC, LANES>(v[i], w + (lo + r) * N, strip0, lane, N);
    else v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.f;
  }
  float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < GROUP_RPT; ++i) max_cols4<false>(m, v[i]);
  *reinterpret_cast<float4*>(&red[rl][lane * 4]) = make_float4(m[0], m[1], m[2], m[3]);
  __syncthreads();
  for (int i = threadIdx.x; i < COLS; i += LANES * RL) {  // slot i: column col_of(i / 4, i % 4)
    float a = red[0][i];
#pragma unroll
    for (int l = 1; l < RL; ++l) a = fmaxf(a, red[l][i]);
    const float s = scale_of(a);
    reinterpret_cast<float*>(scale_s)[i] = s;
    reinterpret_cast<float*>(inv_s)[i] = __frcp_rn(s);
    const int64_t c = col_of<VEC, LANES>(strip0, i / 4, i % 4);
    if (c < N) scales[(int64_t)g * N + c] = s;
  }
  __syncthreads();
  const float4 i4 = inv_s[lane];
  const float inv[4] = {i4.x, i4.y, i4.z, i4.w};
  const float* s = reinterpret_cast<const float*>(scale_s) + lane * 4;  // (read for the few values near a half only)
#pragma unroll
  for (int i = 0; i < GROUP_RPT; ++i) {
    const int r = rl + RL * i;
    if (r < rows) store_codes4<VEC, LANES>(v[i], s, inv, q + (lo + r) * N, strip0, lane, N);
  }
}

template <bool VEC, int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(TALL_WARPS * 32)
quantize_tall_kernel(const float* __restrict__ w, int64_t K, int64_t N, int64_t G, int64_t strips,
                     int8_t* __restrict__ q, float* __restrict__ scales) {
  namespace cg = cooperative_groups;
  constexpr int LANES = TALL_COLS / 4;
  __shared__ float red[2 * TALL_WARPS][TALL_COLS];
  __shared__ float part[TALL_COLS];
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x % LANES, rl = threadIdx.x / LANES;  // column lane, row lane
  const int64_t item = blockIdx.x / CTAS, g = item / strips, strip0 = (item - g * strips) * TALL_COLS;
  const int64_t lo = g * G, hi = lo + G < K ? lo + G : K;
  // row r of the group belongs to row lane r mod (CTAS * 2 * TALL_WARPS) of the cluster
  const int64_t first = lo + (int64_t)cluster.block_rank() * 2 * TALL_WARPS + rl;
  constexpr int64_t kStep = CTAS * 2 * TALL_WARPS;
  float m[4] = {0.f, 0.f, 0.f, 0.f};
  int64_t r = first;
  for (; r + 3 * kStep < hi; r += 4 * kStep) {  // four rows in flight
    float v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) load_cols4<VEC, LANES>(v[i], w + (r + i * kStep) * N, strip0, lane, N);
#pragma unroll
    for (int i = 0; i < 4; ++i) max_cols4<true>(m, v[i]);
  }
  for (; r < hi; r += kStep) {
    float v[4];
    load_cols4<VEC, LANES>(v, w + r * N, strip0, lane, N);
    max_cols4<true>(m, v);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) red[rl][lane + LANES * j] = m[j];
  __syncthreads();
  if (threadIdx.x < TALL_COLS) {
    float a = red[0][threadIdx.x];
#pragma unroll 8
    for (int l = 1; l < 2 * TALL_WARPS; ++l) a = fmaxf(a, red[l][threadIdx.x]);
    part[threadIdx.x] = a;
  }
  cluster.sync();
  if (threadIdx.x < TALL_COLS) {
    float a = 0.f;
#pragma unroll
    for (int b = 0; b < CTAS; ++b) a = fmaxf(a, cluster.map_shared_rank(part, b)[threadIdx.x]);
    red[0][threadIdx.x] = scale_of(a);
  }
  cluster.sync();  // also: no block leaves while another reads its part
  float s[4], inv[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    s[j] = red[0][lane + LANES * j];
    inv[j] = __frcp_rn(s[j]);
  }
  if (cluster.block_rank() == 0 && rl == 0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t c = col_of<VEC, LANES>(strip0, lane, j);
      if (c < N) scales[g * N + c] = s[j];
    }
  }
  r = first;
  for (; r + 3 * kStep < hi; r += 4 * kStep) {
    float v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) load_cols4<VEC, LANES>(v[i], w + (r + i * kStep) * N, strip0, lane, N);
#pragma unroll
    for (int i = 0; i < 4; ++i) store_codes4<VEC, LANES>(v[i], s, inv, q + (r + i * kStep) * N, strip0, lane, N);
  }
  for (; r < hi; r += kStep) {
    float v[4];
    load_cols4<VEC, LANES>(v, w + r * N, strip0, lane, N);
    store_codes4<VEC, LANES>(v, s, inv, q + r * N, strip0, lane, N);
  }
}

// The same in three passes over the whole grid, for matrices whose groups x strips are too few to fill the SMs above: maxima of 128 columns x up to 256 rows of one group merged by atomicMax on the bit
// pattern (non-negative floats order like unsigned integers, so the result does not depend on scheduling), scales in
// place, codes.
constexpr int CHUNK_ROWS = 256, CHUNK_LANES = 8;

struct Quad {
  float v[4];
};

// Four consecutive columns of row r starting at c0; columns >= N read as 0.
__device__ __forceinline__ Quad load_quad(const float* __restrict__ w, int64_t r, int64_t c0, int64_t N, bool vec) {
  Quad o;
  if (vec) {
    const float4 f = *reinterpret_cast<const float4*>(w + r * N + c0);
    o.v[0] = f.x; o.v[1] = f.y; o.v[2] = f.z; o.v[3] = f.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) o.v[j] = (c0 + j < N) ? w[r * N + c0 + j] : 0.f;
  }
  return o;
}

__global__ void __launch_bounds__(256) amax_kernel(const float* __restrict__ w, int64_t K, int64_t N, int64_t G,
                                                    int64_t strips, int64_t chunks_per_group, int vec,
                                                    unsigned int* __restrict__ amax_bits) {
  __shared__ float red[CHUNK_LANES][COLS_PER_BLOCK];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t strip = blockIdx.x % strips, y = blockIdx.x / strips;
  const int64_t g = y / chunks_per_group, ch = y % chunks_per_group;
  const int64_t lo = g * G + ch * CHUNK_ROWS;
  int64_t hi = lo + CHUNK_ROWS;
  if (hi > (g + 1) * G) hi = (g + 1) * G;
  if (hi > K) hi = K;
  const int64_t c0 = strip * COLS_PER_BLOCK + tx * 4;
  float m[4] = {0.f, 0.f, 0.f, 0.f};
  if (c0 < N) {
    for (int64_t r = lo + ty; r < hi; r += CHUNK_LANES) {
      const Quad x = load_quad(w, r, c0, N, vec != 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = fabsf(x.v[j]);
        if (a > m[j]) m[j] = a;  // a NaN never compares greater: skipped, as in the reference
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) red[ty][tx * 4 + j] = m[j];
  __syncthreads();
  if (threadIdx.x < COLS_PER_BLOCK) {
    const int64_t c = strip * COLS_PER_BLOCK + threadIdx.x;
    if (c < N && lo < hi) {
      float a = red[0][threadIdx.x];
#pragma unroll
      for (int l = 1; l < CHUNK_LANES; ++l) a = fmaxf(a, red[l][threadIdx.x]);
      if (a > 0.f) atomicMax(&amax_bits[g * N + c], __float_as_uint(a));
    }
  }
}

__global__ void finalize_scales_kernel(float* __restrict__ scales, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i < n; i += (int64_t)gridDim.x * blockDim.x) scales[i] = scale_of(scales[i]);
}

__global__ void __launch_bounds__(256) quantize_flat_kernel(const float* __restrict__ w, const float* __restrict__ scales,
                                                        int64_t K, int64_t N, int64_t G, int vec,
                                                        int8_t* __restrict__ q) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (vec) {
    const int64_t n4 = K * N / 4;
    for (; i < n4; i += stride) {
      const int64_t e = i * 4, r = e / N, c = e % N;
      const float4 x = *reinterpret_cast<const float4*>(w + e);
      const float4 s = *reinterpret_cast<const float4*>(scales + (r / G) * N + c);
      const uint32_t b0 = (uint32_t)quantize_one(x.x, s.x) & 0xffu, b1 = (uint32_t)quantize_one(x.y, s.y) & 0xffu,
                     b2 = (uint32_t)quantize_one(x.z, s.z) & 0xffu, b3 = (uint32_t)quantize_one(x.w, s.w) & 0xffu;
      *reinterpret_cast<uint32_t*>(q + e) = b0 | (b1 << 8) | (b2 << 16) | (b3 << 24);
    }
  } else {
    const int64_t n = K * N;
    for (; i < n; i += stride) {
      const int64_t r = i / N, c = i % N;
      q[i] = (int8_t)quantize_one(w[i], scales[(r / G) * N + c]);
    }
  }
}

__device__ __forceinline__ uint32_t trunc_bf16(int q, float s) {
  return __float_as_uint(__fmul_rn((float)q, s)) >> 16;
}

// VEC: a lane's eight columns are consecutive (one 8-byte load, one 16-byte store), else 32 apart.
template <bool VEC>
__global__ void __launch_bounds__(256) dequant_kernel(const int8_t* __restrict__ q, const float* __restrict__ scales,
                                                       int64_t K, int64_t N, int64_t G, unsigned strips,
                                                       uint16_t* __restrict__ out) {
  constexpr int RPT = DEQ_ROWS / 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned y = blockIdx.x / strips;
  const int64_t strip0 = (int64_t)(blockIdx.x - y * strips) * DEQ_COLS, r0 = (int64_t)y * DEQ_ROWS;
  auto col = [&](int j) -> int64_t { return VEC ? strip0 + lane * 8 + j : strip0 + lane + 32 * j; };
  uint2 p[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int64_t r = r0 + warp + 8 * i;
    p[i] = make_uint2(0u, 0u);
    if (r >= K) continue;
    if (VEC) {
      if (col(0) < N) p[i] = *reinterpret_cast<const uint2*>(q + r * N + col(0));
    } else {
      uint32_t h[2] = {0u, 0u};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col(j) < N) h[j >> 2] |= (uint32_t)(uint8_t)q[r * N + col(j)] << (8 * (j & 3));
      p[i] = make_uint2(h[0], h[1]);
    }
  }
  float s[8];
  int64_t g_have = -1, g_end = 0;  // the group whose scales are held, and its first row past the end
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int64_t r = r0 + warp + 8 * i;
    if (r >= K) break;
    if (g_have < 0 || r >= g_end) {  // (uniform over the warp)
      g_have = r / G;
      g_end = (g_have + 1) * G;
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = 0.f;
      if (VEC) {
        if (col(0) < N) {
          const float4* sp = reinterpret_cast<const float4*>(scales + g_have * N + col(0));
          const float4 a = sp[0], b = sp[1];
          s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
          s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (col(j) < N) s[j] = scales[g_have * N + col(j)];
      }
    }
    uint32_t h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t word = j < 4 ? p[i].x : p[i].y;
      h[j] = trunc_bf16((int)(int8_t)((word >> (8 * (j & 3))) & 0xffu), s[j]);
    }
    if (VEC) {
      if (col(0) < N)
        *reinterpret_cast<uint4*>(out + r * N + col(0)) =
            make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col(j) < N) out[r * N + col(j)] = (uint16_t)h[j];
    }
  }
}

// Strips that few columns fill, and groups of few rows: the same over one flat list.
template <bool VEC>
__global__ void __launch_bounds__(256) dequant_flat_kernel(const int8_t* __restrict__ q, const float* __restrict__ scales,
                                                           int64_t K, int64_t N, int64_t G, uint16_t* __restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (!VEC) {
    const int64_t n = K * N;
    for (; i < n; i += stride) {
      const int64_t r = i / N, c = i % N;
      out[i] = (uint16_t)trunc_bf16((int)q[i], scales[(r / G) * N + c]);
    }
    return;
  }
  for (const int64_t n8 = K * N / 8; i < n8; i += stride) {
    const int64_t e = i * 8, r = e / N, c = e % N;
    const uint2 p = *reinterpret_cast<const uint2*>(q + e);
    const float* srow = scales + (r / G) * N + c;
    const float4 s0 = *reinterpret_cast<const float4*>(srow), s1 = *reinterpret_cast<const float4*>(srow + 4);
    const float s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    uint32_t h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t word = j < 4 ? p.x : p.y;
      h[j] = trunc_bf16((int)(int8_t)((word >> (8 * (j & 3))) & 0xffu), s[j]);
    }
    *reinterpret_cast<uint4*>(out + e) =
        make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
  }
}

inline unsigned grid_for(int64_t work_items) {
  const int64_t blocks = (work_items + 255) / 256;
  const int64_t cap = 148LL * 32;  // enough blocks in flight to cover HBM latency; the loops stride
  return (unsigned)(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int launch_quantize_passes(const float* w, int64_t K, int64_t N, int64_t G, int8_t* q, float* scales, cudaStream_t s) {
  const int64_t groups = (K + G - 1) / G, strips = (N + COLS_PER_BLOCK - 1) / COLS_PER_BLOCK;
  const int64_t chunks = (G + CHUNK_ROWS - 1) / CHUNK_ROWS;
  ATENIA_CUDA_TRY(cudaMemsetAsync(scales, 0, (size_t)(groups * N) * sizeof(float), s));
  const int vec_w = (N % 4 == 0 && aligned16(w)) ? 1 : 0;
  amax_kernel<<<(unsigned)(strips * groups * chunks), 256, 0, s>>>(w, K, N, G, strips, chunks, vec_w,
                                                                   reinterpret_cast<unsigned int*>(scales));
  count_launch();
  ATENIA_CUDA_TRY(cudaGetLastError());
  finalize_scales_kernel<<<grid_for(groups * N), 256, 0, s>>>(scales, groups * N);
  count_launch();
  ATENIA_CUDA_TRY(cudaGetLastError());
  const int vec_q = (vec_w && aligned16(scales) && (reinterpret_cast<uintptr_t>(q) & 3u) == 0) ? 1 : 0;
  quantize_flat_kernel<<<grid_for(vec_q ? K * N / 4 : K * N), 256, 0, s>>>(w, scales, K, N, G, vec_q, q);
  count_launch();
  return (int)cudaGetLastError();
}

template <bool VEC, int CTAS>
int launch_quantize_tall(const float* w, int64_t K, int64_t N, int64_t G, int8_t* q, float* scales, cudaStream_t s) {
  const int64_t strips = (N + TALL_COLS - 1) / TALL_COLS, items = strips * ((K + G - 1) / G);
  if (items > 0x7fffffffLL / CTAS) return launch_quantize_passes(w, K, N, G, q, scales, s);
  quantize_tall_kernel<VEC, CTAS><<<(unsigned)(items * CTAS), TALL_WARPS * 32, 0, s>>>(w, K, N, G, strips, q, scales);
  count_launch();
  return (int)cudaGetLastError();
}

template <bool VEC, int LANES, int RL>
int launch_quantize_groups(const float* w, int64_t K, int64_t N, int64_t G, int8_t* q, float* scales, cudaStream_t s) {
  const int64_t strips = (N + 4 * LANES - 1) / (4 * LANES), blocks = strips * ((K + G - 1) / G);
  if (blocks > 0x7fffffffLL) return launch_quantize_passes(w, K, N, G, q, scales, s);
  quantize_groups_kernel<VEC, LANES, RL><<<(unsigned)blocks, LANES * RL, 0, s>>>(w, K, N, (int)G, (unsigned)strips, q, scales);
  count_launch();
  return (int)cudaGetLastError();
}

// Where the lines lie (B200, us; the Python call costs about 15, so short ones are all launch):
//   few tall items   a cluster walks K / 256 rows per lane whatever the width.  Eight items or fewer of more than
//                    16384 rows, clusters / three passes: 16384 x 256 19.2 / 24.7, 32768 x 64 31.6 / 25.0, 65536 x 512
//                    112 / 89, 262144 x 128 382 / 89; 16 items: 65536 x 1024 136 / 160
//   blocks per item  8192 x 14336, the cluster taken / clusters of eight / three passes: groups of 256 163 / 836 / 271, of
//                    512 141 / 530 / 268 (one block), of 1024 148 / 279 / 268, of 2048 156 / 201 / 267 (two), of 4096 165 /
//                    165 / 267; 2048 x 4096 by 256 17.4 / 56.4 / 32.1
//   short groups     the groups kernel in blocks no taller than the group needs.  Blocks of 32 rows x 64 columns / of 16 x 64
//                    (groups of 9 to 16) or 8 x 128 (up to 8) / three passes: 4096 x 14336 by 1 668 / 242 / 1049, by 8 105 /
//                    54 / 240, by 16 66 / 51 / 199; 262144 x 32 by 1 205 / 150 / 476, by 8 33.0 / 33.0 / 92.3, by 16 21.3 / 17.2 /
//                    69.3; 300000 x 100 by 8 71 / 37 / 148; narrow and tall, 1048576 x 8 by 128 26.9 / - / 71.9
template <bool VEC>
int launch_quantize(const float* w, int64_t K, int64_t N, int64_t G, int8_t* q, float* scales, cudaStream_t s) {
  const int64_t groups = (K + G - 1) / G;
  if (G > GROUP_ROWS_MAX) {
    const int64_t items = groups * ((N + TALL_COLS - 1) / TALL_COLS);
    if (items <= 8 && G > 16384) return launch_quantize_passes(w, K, N, G, q, scales, s);
    int ctas = G >= 4096 ? 8 : G >= 1024 ? 2 : 1;
    while (ctas < 8 && items * ctas < 256 && G >= ctas * 256) ctas *= 2;  // (fill the SMs with 128 rows a block or more)
    return ctas == 1   ? launch_quantize_tall<VEC, 1>(w, K, N, G, q, scales, s)
           : ctas == 2 ? launch_quantize_tall<VEC, 2>(w, K, N, G, q, scales, s)
           : ctas == 4 ? launch_quantize_tall<VEC, 4>(w, K, N, G, q, scales, s)
                       : launch_quantize_tall<VEC, 8>(w, K, N, G, q, scales, s);
  }
  if (G <= 8) return launch_quantize_groups<VEC, 32, 1>(w, K, N, G, q, scales, s);
  if (G <= 16) return launch_quantize_groups<VEC, 16, 2>(w, K, N, G, q, scales, s);
  if (G <= 32) return launch_quantize_groups<VEC, 16, 4>(w, K, N, G, q, scales, s);
  if (G <= 64) return launch_quantize_groups<VEC, 16, 8>(w, K, N, G, q, scales, s);
  return launch_quantize_groups<VEC, 8, 16>(w, K, N, G, q, scales, s);
}

}  // namespace
}  // namespace atenia

extern "C" {

int atenia_quantize_per_group_i8(const float* w, int64_t K, int64_t N, int64_t group_size, int8_t* q, float* scales,
                                 void* stream) {
  using namespace atenia;
  if (K < 0 || N < 0 || group_size < 0) return ATENIA_ERR_SHAPE;
  if (K == 0 || N == 0) return ATENIA_OK;
  if (!w || !q || !scales) return ATENIA_ERR_NULL;
  const int64_t G = (group_size == 0 || group_size > K) ? K : group_size;
  const int64_t groups = (K + G - 1) / G, strips = (N + COLS_PER_BLOCK - 1) / COLS_PER_BLOCK;
  if (strips * groups * ((G + CHUNK_ROWS - 1) / CHUNK_ROWS) > 0x7fffffffLL || groups > 0x7fffffffLL * 4 / N)
    return ATENIA_ERR_SHAPE;
  const bool vec = N % 4 == 0 && aligned16(w) && (reinterpret_cast<uintptr_t>(q) & 3u) == 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return vec ? launch_quantize<true>(w, K, N, G, q, scales, s) : launch_quantize<false>(w, K, N, G, q, scales, s);
}

int atenia_int8_to_bf16_per_group(const int8_t* q, const float* scales, int64_t K, int64_t N, int64_t group_size,
                                  uint16_t* out_bf16, void* stream) {
  using namespace atenia;
  if (K < 0 || N < 0 || group_size < 0) return ATENIA_ERR_SHAPE;
  if (K == 0 || N == 0) return ATENIA_OK;
  if (!q || !scales || !out_bf16) return ATENIA_ERR_NULL;
  const int64_t G = (group_size == 0 || group_size > K) ? K : group_size;
  const int64_t strips = (N + DEQ_COLS - 1) / DEQ_COLS, chunks = (K + DEQ_ROWS - 1) / DEQ_ROWS;
  if (strips > 0x7fffffffLL / chunks) return ATENIA_ERR_SHAPE;
  const unsigned grid = (unsigned)(strips * chunks);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool vec = N % 8 == 0 && aligned16(out_bf16) && aligned16(scales) && (reinterpret_cast<uintptr_t>(q) & 7u) == 0;
  // strips filled to less than five eighths: the flat walk (262144 rows, strips / flat: 32 columns 27.4 / 14.3 us, 128
  // 29.4 / 22.9, 160 31.3 / 29.4, 192 31.5 / 33.6; 131072 x 264 29.5 / 24.6; unaligned rows gain nothing: x 100 68 / 81);
  // and groups of under 16 rows, whose scales a lane holds for one row in eight (4096 x 14336 by 1 / 8 / 16 72.6 / 64.3,
  // 60.3 / 45.9, 43.2 / 43.9; 300000 x 100 by 8 120 / 109)
  if (vec && (G < 16 || 8 * N <= 5 * DEQ_COLS * strips))
    dequant_flat_kernel<true><<<grid_for(K * N / 8), 256, 0, s>>>(q, scales, K, N, G, out_bf16);
  else if (G < 16)
    dequant_flat_kernel<false><<<grid_for(K * N), 256, 0, s>>>(q, scales, K, N, G, out_bf16);
  else if (vec)
    dequant_kernel<true><<<grid, 256, 0, s>>>(q, scales, K, N, G, (unsigned)strips, out_bf16);
  else
    dequant_kernel<false><<<grid, 256, 0, s>>>(q, scales, K, N, G, (unsigned)strips, out_bf16);
  count_launch();
  return (int)cudaGetLastError();
}

}  // extern "C"
