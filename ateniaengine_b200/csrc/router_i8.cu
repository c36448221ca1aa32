// Router of long bf16 prompts on the int8 tensor cores, with the f64 sums' precision for every input.
//
// The reference accumulates the router logits in f64, and the f64 tensor-core kernel (router_dmma.cu) is bound by the
// f64 pipe and the conversions in front of it: 107 us for 8192 tokens, 64 experts, d = 2048, in which no expert GEMM
// gets far.  Here both operands become integers on a grid of their row's largest magnitude and the products are exact
// (router_digits.cuh has the grids):
//   x[t, :] = 2^(ex - 30) X, four balanced base-256 digits; ex per token and k-range
//   w[e, :] = 2^(ew - 38) W, five digits; made once per set_weights from the layer's copy
//   logit   = 2^(ex + ew - 68) sum_s 256^(7 - s) A_s,  A_s = sum over i + j = s of the digit products, exact in int32
// The eight A_s of 64 experts fill tensor memory; they are put together in f64 (three exact partial sums).
//
// Values off the grid (more than 2^22 below the largest of their k-range: of 2048 normal values there is one in a thousand
// tokens) are not rounded away: a token that may have any is marked while its largest value is looked for, and what its
// digits left out, x - 2^(ex - 30) X, is multiplied by the f32 router rows in f64 and added to its share, value by value.  B200,
// 64 experts of d = 2048, normal activations, kernel without / with this, us: 1300 tokens 19.5 / 21.0, 2048 26.4 / 27.9, 8192
// 44.4 / 46.2.  With a value 2^14 above the rest in every token (a few values a token off the grid) a forward of 8192 tokens
// takes 10 us more and is still below the f64 router's; from 2^18 on, where no model's activations are, it is slower (2^18
// 0.25 ms, all values off the grid 1.3 ms more).
// A layer whose router rows or gate vector are not all on their grid (f32 values that bf16 does not hold) has a row scale
// of NaN: launch_router keeps such a layer on the f64 routers, and a captured launch that meets it after new weights
// computes those rows in f64 here.
//
// CTA = 128 tokens x one k-range of a cluster of 8, 4, 2 or 1; per k-block of 128 the 16 converting warps write the
// four digit planes of the tokens (64 KiB, 128-byte swizzle), TMA brings the five planes of the experts (40 KiB), one
// warp issues twenty M128 x N64 x K32 products per 32 k, plane i of x against plane j of w onto A_(i + j).  The f64
// shares of the k-ranges meet in distributed shared memory in CTA order, then bias, rounding, softmax and top-k by one
// warp per token.
// The shared expert's gate vector is one more row of w.  A token with an infinite or NaN value gets NaN logits, as from
// the f64 sums.  All waits are bounded; a token block whose products did not finish gets NaN logits too.
#include "route_warp.cuh"
#include "router_digits.cuh"
#include "tc_common.cuh"

namespace atenia {
namespace {
using namespace tc;

constexpr int RE = kRouterDigitRows;      // rows of one digit plane of w: experts, the gate vector, zeros
constexpr int RPX = 4, RPW = kRouterDigitPlanes;  // digit planes of x and w
constexpr int RM = 128, RKB = 128;        // tokens per CTA, k per k-block
constexpr int R_STAGES = 2;
constexpr int R_A_PLANE = RM * RKB, R_A_BYTES = RPX * R_A_PLANE;  // 64 KiB
constexpr int R_B_BYTES = RPW * RE * RKB;                         // 40 KiB
constexpr int R_CONV_WARPS = 16, R_THREADS = 64 + R_CONV_WARPS * 32;
constexpr int R_SMEM = R_STAGES * (R_A_BYTES + R_B_BYTES) + 1024;
constexpr int R_PART_LD = RE + 1;  // doubles per token of the shares (odd: lanes hold tokens)
// after the products the stages hold the shares, the logits and the softmax scratch
constexpr int R_LG_OFF = RM * R_PART_LD * 8, R_EXP_OFF = R_LG_OFF + RM * RE * 4;
constexpr int R_NT_MAX = 4;  // tokens that a warp routes at a time
static_assert(R_EXP_OFF + R_THREADS / 32 * R_NT_MAX * R_PART_LD * 8 <= R_STAGES * (R_A_BYTES + R_B_BYTES), "scratch fits the stages");
static_assert(RE == 64 && RPX + RPW - 1 == 8, "tensor memory: eight sums of 64 columns");

struct __align__(8) BarriersR {
  uint64_t full_a[R_STAGES];  // 16 converting warps
  uint64_t full_b[R_STAGES];  // TMA bytes
  uint64_t empty[R_STAGES];   // the MMAs that read the stage are done (commit)
  uint64_t acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t idesc_r(int n) {  // kind::i8: D s32, A = B = s8, K-major, M = 128
  return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(RM >> 4) << 24);
}
// One plane of x (32 bytes of each row) against the five planes of w, plane j onto the sum 64 j columns on.  One block for
// the five: a lane is elected once and the operands stay in uniform registers (see uniform_warp).  `more`: the first four
// sums hold something, `more4`: the last one does.
__device__ __forceinline__ void mma_i8_planes(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t more, uint32_t more4) {
  asm volatile(
      "{\n\t.reg .pred e, p, q;\n\t"
      ".reg .b64 b;\n\t"
      ".reg .b32 d;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t"
      "add.s64 b, %2, %6;\n\tadd.s32 d, %0, 64;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::i8 [d], %1, b, %3, p;\n\t"
      "add.s64 b, b, %6;\n\tadd.s32 d, d, 64;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::i8 [d], %1, b, %3, p;\n\t"
      "add.s64 b, b, %6;\n\tadd.s32 d, d, 64;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::i8 [d], %1, b, %3, p;\n\t"
      "add.s64 b, b, %6;\n\tadd.s32 d, d, 64;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::i8 [d], %1, b, %3, q;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(more), "r"(more4), "n"(RE * RKB / 16)
      : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, int32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
// |n| < 2^51, exact
__device__ __forceinline__ double to_double(long long n) {
  return __longlong_as_double(0x4338000000000000LL + n) - 6755399441055744.0;  // 1.5 * 2^52
}

// Sixteen values of a row -> 16 bytes in each of the four digit planes (top digit first).
__device__ __forceinline__ void digits16(const uint4 (&q)[2], float mul, uint4 (&out)[RPX]) {
  uint32_t p[RPX][4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint32_t w0 = g & 1 ? (g & 2 ? q[1].z : q[0].z) : (g & 2 ? q[1].x : q[0].x);
    const uint32_t w1 = g & 1 ? (g & 2 ? q[1].w : q[0].w) : (g & 2 ? q[1].y : q[0].y);
    uint32_t y[4];
    y[0] = digits_x_bytes(__float2int_rn(bf16lo(w0) * mul));
    y[1] = digits_x_bytes(__float2int_rn(bf16hi(w0) * mul));
    y[2] = digits_x_bytes(__float2int_rn(bf16lo(w1) * mul));
    y[3] = digits_x_bytes(__float2int_rn(bf16hi(w1) * mul));
    const uint32_t a = __byte_perm(y[0], y[1], 0x5140), b = __byte_perm(y[0], y[1], 0x7362);
    const uint32_t c = __byte_perm(y[2], y[3], 0x5140), d = __byte_perm(y[2], y[3], 0x7362);
    p[3][g] = __byte_perm(a, c, 0x5410);
    p[2][g] = __byte_perm(a, c, 0x7632);
    p[1][g] = __byte_perm(b, d, 0x5410);
    p[0][g] = __byte_perm(b, d, 0x7632);
  }
#pragma unroll
  for (int i = 0; i < RPX; ++i) out[i] = make_uint4(p[i][0], p[i][1], p[i][2], p[i][3]);
}

// What the digits of one token left out of x[k_begin, k_end), times the rows of w; a row that the planes do not hold (off0, off1;
// w_off: there are any) times all of x.  One warp, lane l rows l and l + 32; values are taken in the order of k.  (Short code: it
// is seldom run, so every line of it is fetched anew.)
__device__ __noinline__ double2 left_out(const __nv_bfloat16* __restrict__ x, int k_begin, int k_end, int ex,
                                         const float* __restrict__ w_router, const float* __restrict__ gate_vec, int E, int d, bool off0,
                                         bool off1, bool w_off, int lane) {
  auto row_of = [&](int e) { return e < E ? w_router + (size_t)e * d : e == E ? gate_vec : nullptr; };
  const float *row0 = row_of(lane), *row1 = row_of(lane + 32);
  // (in f64: a small value next to a huge one would leave the range of f32 on the grid's scale)
  const double mul = __longlong_as_double((long long)(30 - ex + 1023) << 52), unit = __longlong_as_double((long long)(ex - 30 + 1023) << 52);
  const uint32_t edge = digits_x_edge(ex);  // below it a value may be off the grid
  auto low = [&](uint32_t bits) { return bits != 0 && bits < edge; };
  constexpr int U = 4;  // vectors of a lane in flight
  double2 sum = make_double2(0.0, 0.0);
#pragma unroll 1
  for (int k0 = k_begin; k0 < k_end; k0 += U * 256) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * 256 + lane * 8;
      q[u] = k < k_end ? *reinterpret_cast<const uint4*>(x + k) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll 1
    for (int u = 0; u < U; ++u) {
      const uint4 own = q[0];
#pragma unroll
      for (int n = 1; n < U; ++n) q[n - 1] = q[n];
      const int ku = k0 + u * 256;
      const uint32_t ow[4] = {own.x, own.y, own.z, own.w};
      bool some = w_off;
#pragma unroll
      for (int j = 0; j < 4; ++j) some = some || low(ow[j] & 0x7fffu) || low(ow[j] >> 16 & 0x7fffu);
      for (unsigned todo = __ballot_sync(0xffffffffu, some && ku + lane * 8 < k_end); todo; todo &= todo - 1) {
        const int from = __ffs(todo) - 1, k = ku + from * 8;
        // eight values: lane j (j < 8) makes its own ready
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t v = __shfl_sync(0xffffffffu, ow[j], from);
          if ((lane >> 1 & 3) == j) word = v;
        }
        const double v = lane & 1 ? bf16hi(word) : bf16lo(word), f = v * mul, left = (f - rint(f)) * unit;
        unsigned which = __ballot_sync(0xffffffffu, lane < 8 && (w_off || left != 0.0));
        if (__popc(which) > 2) {  // a token of many: all eight, their weights in flight together
          float w0[8], w1[8];
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 a = row0 ? *reinterpret_cast<const float4*>(row0 + k + j) : z, b = row1 ? *reinterpret_cast<const float4*>(row1 + k + j) : z;
            w0[j] = a.x, w0[j + 1] = a.y, w0[j + 2] = a.z, w0[j + 3] = a.w;
            w1[j] = b.x, w1[j + 1] = b.y, w1[j + 2] = b.z, w1[j + 3] = b.w;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const double vj = __shfl_sync(0xffffffffu, v, j), lj = __shfl_sync(0xffffffffu, left, j);
            sum.x = fma(off0 ? vj : lj, (double)w0[j], sum.x);
            sum.y = fma(off1 ? vj : lj, (double)w1[j], sum.y);
          }
          continue;
        }
        for (; which; which &= which - 1) {
          const int j = __ffs(which) - 1;
          const double vj = __shfl_sync(0xffffffffu, v, j), lj = __shfl_sync(0xffffffffu, left, j);
          if (row0) sum.x = fma(off0 ? vj : lj, (double)row0[k + j], sum.x);
          if (row1) sum.y = fma(off1 ? vj : lj, (double)row1[k + j], sum.y);
        }
      }
    }
  }
  return sum;
}

template <int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(R_THREADS, 1)
router_i8_kernel(RouterArgs a, const __grid_constant__ CUtensorMap tmap_w, const double* __restrict__ w_scale) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ BarriersR bars;
  __shared__ int row_exp[RM];  // ex of a token's k-range; kBad: a value is not finite
  __shared__ bool row_off[RM];  // ... a value may be off the grid
  __shared__ int32_t idx_s[R_THREADS / 32][R_NT_MAX][kMaxK];
  __shared__ float w_s[R_THREADS / 32][R_NT_MAX][kMaxK];
  constexpr int kBad = 1 << 20;
  constexpr int R_NT = CTAS >= 8 ? 1 : CTAS == 4 ? 2 : R_NT_MAX;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t b_base = smem_base + R_STAGES * R_A_BYTES;
  volatile int* abort_flag = &bars.abort_flag;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = blockIdx.x % CTAS, t0 = blockIdx.x / CTAS * RM;
  const int d = a.d, E = a.E;
  // k-blocks of this CTA
  const int all_kb = (d + RKB - 1) / RKB, per = (all_kb + CTAS - 1) / CTAS;
  const int kb0 = rank * per < all_kb ? rank * per : all_kb, nkb = (kb0 + per < all_kb ? kb0 + per : all_kb) - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < R_STAGES; ++s) {
      mbar_init(smem_u32(&bars.full_a[s]), R_CONV_WARPS);
      mbar_init(smem_u32(&bars.full_b[s]), 1);
      mbar_init(smem_u32(&bars.empty[s]), 1);
    }
    mbar_init(smem_u32(&bars.acc_full), 1);
    bars.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&bars.tmem_base))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars.tmem_base;

  if (warp == 0) {
    // ================= TMA: the experts' digits =================
    bool ok = true;
    uint32_t armed = 0;
    int i = 0;
    for (; ok && i < nkb; ++i) {
      const int s = i % R_STAGES;
      if (!mbar_wait(smem_u32(&bars.empty[s]), ((i / R_STAGES) & 1u) ^ 1u, abort_flag)) {
        if (lane == 0) report_error(a.err, ATENIA_ERR_DEVICE_TIMEOUT, 3000 + s);
        *abort_flag = 1;
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const uint32_t full = smem_u32(&bars.full_b[s]), dst = b_base + s * R_B_BYTES;
      mbar_expect_tx_one(full, R_B_BYTES);
      tma_load_2d_one(dst, &tmap_w, full, (kb0 + i) * RKB, 0);
      tma_load_2d_one(dst + R_B_BYTES / 2, &tmap_w, full, (kb0 + i) * RKB, RPW * RE / 2);
      armed |= 1u << s;
    }
    if (*abort_flag && lane == 0) {  // copies in flight land before the memory is used for anything else
      for (int s = 0; s < R_STAGES; ++s) {
        if (!(armed & (1u << s))) continue;
        const int last = (i - 1) - ((i - 1 - s) % R_STAGES + R_STAGES) % R_STAGES;  // last k-block of this stage
        for (uint32_t n = 0; n < (1u << 20); ++n)
          if (mbar_try_wait(smem_u32(&bars.full_b[s]), (last / R_STAGES) & 1u)) break;
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer =================
    bool ok = true;
    for (int i = 0; ok && i < nkb; ++i) {
      const int s = i % R_STAGES;
      const uint32_t phase = (i / R_STAGES) & 1u;
      if (!mbar_wait(smem_u32(&bars.full_b[s]), phase, abort_flag) || !mbar_wait(smem_u32(&bars.full_a[s]), phase, abort_flag)) {
        if (lane == 0) report_error(a.err, ATENIA_ERR_DEVICE_TIMEOUT, 3010 + s);
        *abort_flag = 1;
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t sa = smem_base + s * R_A_BYTES;
      const uint32_t sb = b_base + s * R_B_BYTES;
#pragma unroll
      for (int k = 0; k < RKB / 32; ++k) {
        const uint32_t more = (i > 0 || k > 0) ? 1u : 0u;
#pragma unroll
        for (int p = 0; p < RPX; ++p) {
          // (one shape and one accumulator per sum: only such products are sure to follow one another in order)
          mma_i8_planes(tmem_base + RE * p, make_smem_desc(sa + p * R_A_PLANE) + 2 * k, make_smem_desc(sb) + 2 * k, idesc_r(RE),
                        (more || p > 0) ? 1u : 0u, more);
        }
      }
      tc_commit_one(smem_u32(&bars.empty[s]));
    }
    if (ok && nkb > 0) tc_commit_one(smem_u32(&bars.acc_full));
  } else {
    // ================= converting warps, then the epilogue =================
    const int cw = warp - 2;
    // eight lanes cover the 128 k of a row, a warp four rows, the 16 warps 64 rows: two rows per lane
    const int c = lane & 7;
    const __nv_bfloat16* src[2];
    bool in[2];
    int row[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      row[h] = h * 64 + cw * 4 + (lane >> 3);
      in[h] = t0 + row[h] < a.T;
      src[h] = static_cast<const __nv_bfloat16*>(a.x) + (size_t)(in[h] ? t0 + row[h] : 0) * d + c * 16;
    }
    auto load = [&](uint4 (&q)[2][2], int i) {
      const int k = (kb0 + i) * RKB;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        q[h][0] = q[h][1] = make_uint4(0, 0, 0, 0);
        if (in[h] && i < nkb && k + c * 16 < d) {  // (d is a multiple of 16)
          const uint4* p = reinterpret_cast<const uint4*>(src[h] + k);
          q[h][0] = p[0];
          q[h][1] = p[1];
        }
      }
    };
    // largest and smallest (but zeros) magnitude of each row over the k-range: bf16 bit patterns without the sign order like
    // integers
    uint32_t m[2] = {0u, 0u}, key[2] = {0x7fff7fffu, 0x7fff7fffu};
    for (int i = 0; i < nkb; i += 4) {
      uint4 q[4][2][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) load(q[j], i + j);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const uint32_t w[4] = {q[j][h][v].x, q[j][h][v].y, q[j][h][v].z, q[j][h][v].w};
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const uint32_t w0 = w[e] & 0x7fff7fffu, w1 = w[e + 1] & 0x7fff7fffu;
              m[h] = __vimax3_u16x2(m[h], w0, w1);
              key[h] = __vimin3_s16x2(key[h], digits_keys(w0), digits_keys(w1));
            }
          }
    }
    float mul[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t v = max(m[h] & 0xffffu, m[h] >> 16), kk = key[h];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
        kk = __vmins2(kk, __shfl_xor_sync(0xffffffffu, kk, o));
      }
      const int ex = digits_x_exponent(v);  // |x| < 2^ex
      const bool bad = v >= 0x7f80u;
      const bool off = !bad && digits_x_off_grid(digits_of_key(__vmins2(kk, kk >> 16) & 0xffffu), ex);
      if (c == 0) {
        row_exp[row[h]] = bad ? kBad : ex;
        row_off[row[h]] = off;
      }
      mul[h] = bad ? 0.f : __uint_as_float((uint32_t)(30 - ex + 127) << 23);
    }
    bool ok = true;
    uint4 cur[2][2], nxt[2][2];
    load(cur, 0);
    for (int i = 0; i < nkb; ++i) {
      const int s = i % R_STAGES;
      load(nxt, i + 1);
      if (!mbar_wait(smem_u32(&bars.empty[s]), ((i / R_STAGES) & 1u) ^ 1u, abort_flag)) {
        if (lane == 0) report_error(a.err, ATENIA_ERR_DEVICE_TIMEOUT, 3020 + s);
        *abort_flag = 1;
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      uint8_t* stage = smem + s * R_A_BYTES;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint4 dg[RPX];
        digits16(cur[h], mul[h], dg);
        uint8_t* dst = stage + row[h] * RKB + ((c ^ (row[h] & 7)) << 4);
#pragma unroll
        for (int p = 0; p < RPX; ++p) *reinterpret_cast<uint4*>(dst + p * R_A_PLANE) = dg[p];
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars.full_a[s]));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        cur[h][0] = nxt[h][0];
        cur[h][1] = nxt[h][1];
      }
    }
    if (ok && nkb > 0) {
      ok = mbar_wait(smem_u32(&bars.acc_full), 0, abort_flag);
      if (!ok) {
        if (lane == 0) report_error(a.err, ATENIA_ERR_DEVICE_TIMEOUT, 3030);
        *abort_flag = 1;
      }
    }
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    asm volatile("bar.sync 1, %0;" ::"n"(R_CONV_WARPS * 32) : "memory");  // row_exp, row_off; nobody writes a stage any more
    // a lane holds a token (row of the accumulators), a warp 16 experts of its lane quarter
    const int t = (warp & 3) * 32 + lane, e0 = (cw >> 2) * 16;
    const int ex = row_exp[t];
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    const double rs = (ex == kBad || !ok) ? nan : __longlong_as_double((long long)(ex + 1023) << 52);
    double* part = reinterpret_cast<double*>(smem) + (size_t)t * R_PART_LD;
    const uint32_t ta = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    bool w_off = false;  // a row of w that its planes do not hold
#pragma unroll 1
    for (int e = e0; e < e0 + 16; e += 8) {
      int32_t A[8][8];
      if (ok && nkb > 0) {
#pragma unroll
        for (int s = 0; s < 8; ++s) tc_ld8(ta + s * RE + e, A[s]);
        tc_ld_wait();
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        double v = 0.0;
        if (ok && nkb > 0) {
          const int32_t level[8] = {A[0][j], A[1][j], A[2][j], A[3][j], A[4][j], A[5][j], A[6][j], A[7][j]};
          long long p[3];
          digits_fold(level, p);
          v = fma(to_double(p[2]), 0x1p-40, fma(to_double(p[1]), 0x1p-24, to_double(p[0])));
        }
        const double ws = w_scale[e + j];
        w_off = w_off || isnan(ws);
        part[e + j] = v * rs * ws;
      }
    }
    // what the digits left out, once the shares are written: does any token or row of w have some?
    int some;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                 : "=r"(some) : "r"((int)(w_off || row_off[t])), "n"(R_CONV_WARPS * 32) : "memory");
    if (some && ok) {
      const bool off0 = isnan(w_scale[lane]), off1 = isnan(w_scale[lane + 32]);
      w_off = __any_sync(0xffffffffu, off0 || off1);
      for (int r = cw; r < RM; r += R_CONV_WARPS) {
        if (!(row_off[r] || w_off) || row_exp[r] == kBad || t0 + r >= a.T) continue;
        const double2 v = left_out(static_cast<const __nv_bfloat16*>(a.x) + (size_t)(t0 + r) * d, kb0 * RKB, min(d, (kb0 + nkb) * RKB), row_exp[r],
                                   a.w_router, a.gate_vec, E, d, off0, off1, w_off, lane);
        double* share = reinterpret_cast<double*>(smem) + (size_t)r * R_PART_LD + lane;
        share[0] = off0 ? v.x : share[0] + v.x;
        share[32] = off1 ? v.y : share[32] + v.y;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  // ================= tokens rank * (128 / CTAS) ... of the block =================
  constexpr int kMine = RM / CTAS;
  float* lg = reinterpret_cast<float*>(smem + R_LG_OFF);
  const bool gate = a.gate_vec != nullptr && a.gate_scale != nullptr;  // row E of w
  constexpr int U = 16 / CTAS < 8 ? 16 / CTAS : 8;  // logits of a thread whose shares are on their way together
  for (int i0 = threadIdx.x; i0 < kMine * RE; i0 += U * R_THREADS) {
    double v[U][CTAS];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * R_THREADS, mt = i / RE, e = i - mt * RE, t = rank * kMine + mt;
      if (i >= kMine * RE) continue;
      const uint32_t mine = smem_base + (uint32_t)(t * R_PART_LD + e) * 8;
#pragma unroll
      for (int q = 0; q < CTAS; ++q) {
        uint32_t theirs;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(q));
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[u][q]) : "r"(theirs) : "memory");
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * R_THREADS, mt = i / RE, e = i - mt * RE, my = t0 + rank * kMine + mt;
      if (i >= kMine * RE || my >= a.T || !(e < E || (e == E && gate))) continue;
      double sum = 0.0;
#pragma unroll
      for (int q = 0; q < CTAS; ++q) sum += v[u][q];
      if (e == E) {
        a.gate_scale[my] = (float)(1.0 / (1.0 + exp(-sum)));
      } else {
        if (a.bias) sum += (double)a.bias[e];  // the bias joins the f64 sum before the rounding to f32
        const float f = (float)sum;
        lg[mt * RE + e] = f;
        if (a.logits) a.logits[(size_t)my * E + e] = f;
      }
    }
  }
  // (waited for at the end: no CTA leaves while another may read its shares)
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  __syncthreads();
  double* exps = reinterpret_cast<double*>(smem + R_EXP_OFF) + warp * R_NT * R_PART_LD;
  for (int m0 = warp * R_NT; m0 < kMine; m0 += R_THREADS / 32 * R_NT) {
    const int my = t0 + rank * kMine + m0;
    bool valid[R_NT];
    int rc[R_NT];
#pragma unroll
    for (int j = 0; j < R_NT; ++j) valid[j] = m0 + j < kMine && my + j < a.T;
    route_many_warp<RE / 32, R_NT>(lg + m0 * RE, RE, valid, E, a.k, a.renormalize, lane, idx_s[warp], w_s[warp], exps,
                                   R_PART_LD, rc);
#pragma unroll
    for (int j = 0; j < R_NT; ++j) {
      if (!valid[j]) continue;
      if (rc[j] && lane == 0) report_error(a.err, rc[j], 1006);
      if (lane < a.k) {  // (an error keeps downstream kernels in bounds)
        a.topk_idx[(size_t)(my + j) * a.k + lane] = rc[j] ? lane : idx_s[warp][j][lane];
        a.topk_w[(size_t)(my + j) * a.k + lane] = rc[j] ? 0.f : w_s[warp][j][lane];
      }
    }
    __syncwarp();
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

// One block per row of w: experts, then the gate vector (if given), then rows of zeros.
__global__ void __launch_bounds__(256) router_digits_kernel(const float* __restrict__ router, const float* __restrict__ gate,
                                                            int E, int d, int8_t* __restrict__ planes,
                                                            double* __restrict__ scale) {
  __shared__ float red[8];
  const int e = blockIdx.x;
  const float* row = e < E ? router + (size_t)e * d : (e == E ? gate : nullptr);
  float m = 0.f;
  bool bad = false;
  for (int k = threadIdx.x; row && k < d; k += 256) {
    const float v = fabsf(row[k]);
    bad = bad || !(v <= 3.402823466e38f);
    m = fmaxf(m, v);
  }
  if (bad) m = __int_as_float(0x7f800000);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = red[0];
  for (int i = 1; i < 8; ++i) m = fmaxf(m, red[i]);
  const bool finite = m <= 3.402823466e38f;
  const int ew = finite && m > 0.f ? ilogbf(m) + 1 : 0;  // m < 2^ew
  const double mul = ldexp(1.0, 38 - ew);
  bool off = !finite;
  for (int k = threadIdx.x; row && k < d; k += 256) {
    const double v = (double)row[k] * mul;
    off = off || v != rint(v);
  }
  off = __syncthreads_or(off);
  // NaN: the row has values that are not finite or off the grid, and its planes are zero
  if (threadIdx.x == 0) scale[e] = off ? __longlong_as_double(0x7ff8000000000000LL) : ldexp(1.0, ew - 28);
  for (int k = threadIdx.x; k < d; k += 256) {
    long long W = row && !off ? __double2ll_rn((double)row[k] * mul) : 0;
#pragma unroll
    for (int p = RPW - 1; p >= 0; --p) planes[((size_t)p * RE + e) * d + k] = digits_w_next(W);
  }
}

template <int CTAS>
int launch_form(const RouterArgs& a, cudaStream_t s) {
  static bool attr_set[kMaxDevices] = {};
  if (first_use_on_current_device(attr_set))
    ATENIA_CUDA_TRY(cudaFuncSetAttribute(router_i8_kernel<CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, R_SMEM));
  router_i8_kernel<CTAS><<<(a.T + RM - 1) / RM * CTAS, R_THREADS, R_SMEM, s>>>(a, *a.digit_map, a.digit_scale);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_router_digits(const float* router, const float* gate, int E, int d, int8_t* planes, double* scale, cudaStream_t s) {
  router_digits_kernel<<<RE, 256, 0, s>>>(router, gate, E, d, planes, scale);
  count_launch();
  return (int)cudaGetLastError();
}

int launch_router_i8(const RouterArgs& a, cudaStream_t s) {
  if (a.T <= 0) return ATENIA_OK;
  if (a.x_is_f32 || !a.digit_map || !a.digit_scale || a.k > kMaxK || a.E > RE || (a.gate_vec && a.E == RE) || a.d % 16 != 0 || a.d > kRouterDigitMaxK)
    return ATENIA_ERR_UNSUPPORTED;
  const int tiles = (a.T + RM - 1) / RM;
  int rc;
  if (tiles <= 14) rc = launch_form<8>(a, s);
  else if (tiles <= 34) rc = launch_form<4>(a, s);
  else if (tiles <= 72) rc = launch_form<2>(a, s);
  else rc = launch_form<1>(a, s);
  count_launch();
  count_tcgen05_launch();
  return rc;
}

}  // namespace atenia
