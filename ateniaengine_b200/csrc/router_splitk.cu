// Router for batches that do not fill the SMs with whole tokens: the d-long dot products are cut over a cluster.
//
// One cluster of eight (or four, or one) CTAs takes eight tokens.  Slice s of the k-range belongs to CTA s mod 8 of the
// cluster and to one of its warp rows; the products are the f64 tensor-core products of router_dmma.cu (same fragments,
// same permuted summation index).  The warps' partial sums are added in shared memory, the CTAs' through distributed
// shared memory, CTA by CTA; the tokens of the block are finished (bias, rounding to f32, softmax, top-k) by one warp
// each, spread over the CTAs.  Every order of additions is fixed.
//
// Bound by latency: two loads deep (the router rows are the layer's own, so they are requested before chain_wait()), the
// products, two barriers, one softmax; from a few hundred tokens on by the f64 products.  B200, us, a form that left the
// slices in a workspace for the last CTA to add (up to 128 tokens) or one CTA per eight tokens (above) / this one:
//   8 experts, d 4096    8 tokens 8.0 / 4.3, 128 12.2 / 4.7, 256 7.5 / 5.0, 512 7.5 / 5.8, 2048 16.3 / 12.0
//   64 experts, d 2048   8 tokens 12.1 / 6.6, 64 12.5 / 6.8, 256 18.3 / 8.5, 512 19.2 / 12.1, 2048 38.9 / 30.7
//   128 experts, d 2048  8 tokens 18.0 / 9.3, 256 34.6 / 13.3, 512 34.6 / 20.3, 2048 70.1 / 58.7
// Between 513 and 1184 tokens one CTA per eight tokens (router_dmma.cu) is as fast (64 experts, 1000 tokens 19.6 / 22 and
// more), above 2368 its form of 16 tokens per CTA is (4096 tokens 54 / 58), and for a router matrix of 4096 words or less
// it needs no cluster barriers (8 experts, d 512, 64 tokens 3.6 / 4.3); nor does one of under 32768 words above 128 tokens
// (forwards of 16 INT8 experts of d 1024, 256 / 500 tokens 84.5 / 86.5, 90.5 / 92.7).  Clusters of one fill the register files, which keeps a
// shared expert's GEMMs off the SMs (64 INT8 experts, f32, 1500 tokens 432 / 446 a forward): not beside one.  router_splitk_pays.
#include "dmma.cuh"
#include "route_warp.cuh"

namespace atenia {
namespace {

constexpr int kSkTok = 8;   // tokens per cluster
constexpr int kSkWarps = 8;
constexpr int kSkFewTokens = 512;
constexpr int kSkSteps = 4;  // steps of 32 k whose router rows are in flight together

template <int E_T, bool XF, int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(kSkWarps * 32, 2)
router_splitk_kernel(RouterArgs a, int kw) {
  constexpr int NT = E_T / 8, NTW = NT < 2 ? NT : 2;  // 8-expert tiles, of which a warp owns NTW
  constexpr int NW_N = NT / NTW, NW_K = kSkWarps / NW_N;
  static_assert(NW_N * NW_K == kSkWarps, "warp arrangement");
  constexpr int XW = XF ? 8 : 4;  // 32-bit words of a lane's eight x values
  __shared__ double part_s[kSkWarps][NTW][32][2];
  __shared__ double gpart_s[kSkWarps][kSkTok];
  __shared__ double sum_s[kSkTok][E_T + 1];  // this CTA's share of the logits; column E_T: of the gate
  constexpr int kMine = kSkTok / CTAS;  // tokens that a CTA finishes: rank, rank + CTAS, ...
  __shared__ float lg_s[kMine][E_T];
  __shared__ double exps_s[kMine][E_T];
  __shared__ int32_t idx_s[kMine][kMaxK];
  __shared__ float w_s[kMine][kMaxK];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ngrp = warp % NW_N, kslice = warp / NW_N;
  const int r = lane >> 2, c = lane & 3;
  const int rank = blockIdx.x % CTAS;
  const int t0 = blockIdx.x / CTAS * kSkTok;
  const int d = a.d, E = a.E;
  const int s0 = (kslice * CTAS + rank) * kw;
  const int k_begin = s0 < d ? s0 : d, k_end = k_begin + kw < d ? k_begin + kw : d;
  const int tg = t0 + r;

  double acc[NTW][2], gacc = 0.0;
#pragma unroll
  for (int j = 0; j < NTW; ++j) acc[j][0] = acc[j][1] = 0.0;
  uint32_t wq[kSkSteps][NTW][8], xq[2][XW];  // raw words: router rows of four steps, x of two
  auto fetch_w = [&](int kb) {
#pragma unroll
    for (int i = 0; i < kSkSteps; ++i) {
      const int k = kb + 32 * i + c * 8;
      const bool k_ok = k < k_end;  // d and kw are multiples of 8: a lane's values are all in or all out
#pragma unroll
      for (int j = 0; j < NTW; ++j) {
        const int e = (ngrp * NTW + j) * 8 + r;
        zero_words(wq[i][j]);
        if (k_ok && e < E) ld_words<8, true>(wq[i][j], a.w_router + (size_t)e * d + k);
      }
    }
  };
  auto fetch_x = [&](auto BUF, int kb) {
    constexpr int b = decltype(BUF)::value;
    const int k = kb + c * 8;
    zero_words(xq[b]);
    if (k < k_end && tg < a.T) {
      if (XF) ld_words<XW, false>(xq[b], static_cast<const float*>(a.x) + (size_t)tg * d + k);
      else ld_words<XW, false>(xq[b], static_cast<const __nv_bfloat16*>(a.x) + (size_t)tg * d + k);
    }
  };
  auto multiply = [&](auto STEP) {
    constexpr int i = decltype(STEP)::value, b = i & 1;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const double xv = x_elem<XF>(xq[b], j);
#pragma unroll
      for (int jt = 0; jt < NTW; ++jt) dmma884(acc[jt], xv, (double)__uint_as_float(wq[i][jt][j]));
    }
  };
  chain_next();
  fetch_w(k_begin);  // (the layer's copies: no kernel writes them)
  // the dot product with the shared expert's gate vector: steps of 32 k dealt over all warps of the cluster
  const int g_begin = (warp * CTAS + rank) * 32 + c * 8;
  uint32_t gq[8];
  zero_words(gq);
  if (a.gate_vec && g_begin < d) ld_words<8, true>(gq, a.gate_vec + g_begin);
  chain_wait();
  for (int kb = k_begin; kb < k_end; kb += 32 * kSkSteps) {
    if (kb != k_begin) fetch_w(kb);
    fetch_x(Int<0>{}, kb);
    fetch_x(Int<1>{}, kb + 32);
    multiply(Int<0>{});  // (past k_end every word is zero)
    fetch_x(Int<0>{}, kb + 64);
    multiply(Int<1>{});
    if (kb + 64 < k_end) {  // (uniform over the warp)
      fetch_x(Int<1>{}, kb + 96);
      multiply(Int<2>{});
      multiply(Int<3>{});
    }
  }
#pragma unroll
  for (int jt = 0; jt < NTW; ++jt) {
    part_s[warp][jt][lane][0] = acc[jt][0];
    part_s[warp][jt][lane][1] = acc[jt][1];
  }
  if (a.gate_vec) {
    for (int k = g_begin; k < d; k += 32 * CTAS * kSkWarps) {
      uint32_t xg[XW];
      zero_words(xg);
      if (tg < a.T) {
        if (XF) ld_words<XW, false>(xg, static_cast<const float*>(a.x) + (size_t)tg * d + k);
        else ld_words<XW, false>(xg, static_cast<const __nv_bfloat16*>(a.x) + (size_t)tg * d + k);
      }
      if (k != g_begin) ld_words<8, true>(gq, a.gate_vec + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) gacc = fma((double)__uint_as_float(gq[j]), x_elem<XF>(xg, j), gacc);
    }
    __syncwarp();
    // the four lanes of a row hold the k-quarters of its dot product: fold them (fixed tree)
    gacc += __shfl_xor_sync(0xffffffffu, gacc, 1);
    gacc += __shfl_xor_sync(0xffffffffu, gacc, 2);
    if (c == 0) gpart_s[warp][r] = gacc;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kSkTok * E_T; i += kSkWarps * 32) {
    const int t = i / E_T, e = i - t * E_T;
    const int nt = e >> 3, col = e & 7, og = nt / NTW, jt = nt - og * NTW;
    double v = 0.0;
#pragma unroll
    for (int ks = 0; ks < NW_K; ++ks) v += part_s[ks * NW_N + og][jt][t * 4 + (col >> 1)][col & 1];
    sum_s[t][e] = v;
  }
  if (a.gate_vec && threadIdx.x < kSkTok) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < kSkWarps; ++w) v += gpart_s[w][threadIdx.x];
    sum_s[threadIdx.x][E_T] = v;
  }
  __syncwarp();  // (.aligned: the lanes of a warp arrive together)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  // this CTA's tokens: the shares of their logits in CTA order, then the bias, then the rounding to f32
  for (int i = threadIdx.x; i < kMine * (E_T + 1); i += kSkWarps * 32) {
    const int m = i / (E_T + 1), e = i - m * (E_T + 1), t = m * CTAS + rank, my = t0 + t;
    if (my >= a.T || !(e < E || (e == E_T && a.gate_vec && a.gate_scale))) continue;
    const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(&sum_s[t][e]));
    double v[CTAS], sum = 0.0;
#pragma unroll
    for (int q = 0; q < CTAS; ++q) {
      uint32_t theirs;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(q));
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[q]) : "r"(theirs) : "memory");
    }
#pragma unroll
    for (int q = 0; q < CTAS; ++q) sum += v[q];
    if (e == E_T) {
      a.gate_scale[my] = (float)(1.0 / (1.0 + exp(-sum)));
    } else {
      if (a.bias) sum += (double)a.bias[e];  // the bias joins the f64 sum before the rounding to f32
      const float f = (float)sum;
      lg_s[m][e] = f;
      if (a.logits) a.logits[(size_t)my * E + e] = f;
    }
  }
  // (waited for at the end: no CTA leaves while another may read its shares)
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  __syncthreads();
  const int my = t0 + warp * CTAS + rank;  // one warp per token
  if (warp < kMine && my < a.T) {
    const int rc = route_one_warp<(E_T + 31) / 32>(lg_s[warp], E, a.k, a.renormalize, lane, idx_s[warp], w_s[warp], exps_s[warp]);
    if (rc) {
      if (lane == 0) report_error(a.err, rc, 1004);
      if (lane < a.k) {  // keep downstream kernels in bounds
        idx_s[warp][lane] = lane;
        w_s[warp][lane] = 0.f;
      }
    }
    __syncwarp();
    if (lane < a.k) {
      a.topk_idx[(size_t)my * a.k + lane] = idx_s[warp][lane];
      a.topk_w[(size_t)my * a.k + lane] = w_s[warp][lane];
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int E_T, int CTAS>
int launch_form(const RouterArgs& a, bool chained, cudaStream_t s) {
  constexpr int NT = E_T / 8, NTW = NT < 2 ? NT : 2;
  constexpr int kSlices = CTAS * (kSkWarps / (NT / NTW));
  const int kw = ((a.d + kSlices - 1) / kSlices + 31) / 32 * 32;  // k-range of a slice: whole steps of 32
  const dim3 grid((a.T + kSkTok - 1) / kSkTok * CTAS), block(kSkWarps * 32);
  if (a.x_is_f32) return launch_chained(chained, router_splitk_kernel<E_T, true, CTAS>, grid, block, 0, s, a, kw);
  return launch_chained(chained, router_splitk_kernel<E_T, false, CTAS>, grid, block, 0, s, a, kw);
}

// CTAs per cluster: as many as let every cluster run at once (two CTAs per SM).  From 1185 tokens on a cluster of one, a
// plain launch (see router_dmma.cu).
template <int E_T>
int launch_one(const RouterArgs& a, cudaStream_t s) {
  if (a.T <= 256) return launch_form<E_T, 8>(a, a.chained, s);
  if (a.T <= kSkFewTokens) return launch_form<E_T, 4>(a, a.chained, s);
  return launch_form<E_T, 1>(a, false, s);
}

}  // namespace

bool router_splitk_pays(int T, int E, int d, bool beside) {
  const int64_t words = (int64_t)E * d;
  if (d % 16 != 0 || words <= 4096) return false;
  if (T <= kSkFewTokens) return T <= 128 || words >= 1 << 15;
  return !beside && T > 8 * 148 && T <= 16 * 148;
}

int launch_router_splitk(const RouterArgs& a, cudaStream_t s) {
  if (a.T <= 0) return ATENIA_OK;
  if (a.k > kMaxK || a.E > 128 || a.d % 16 != 0) return ATENIA_ERR_UNSUPPORTED;
  int rc;
  if (a.E <= 8) rc = launch_one<8>(a, s);
  else if (a.E <= 16) rc = launch_one<16>(a, s);
  else if (a.E <= 32) rc = launch_one<32>(a, s);
  else if (a.E <= 64) rc = launch_one<64>(a, s);
  else rc = launch_one<128>(a, s);
  count_launch();
  return rc;
}

}  // namespace atenia
