// Softmax + top-k of one token by one warp, shared by the router kernels.
#pragma once
#include "common.cuh"

namespace atenia {

constexpr int kMaxK = 8;

// Softmax + top-k for one token by one warp.  `lg` holds E f32 logits in shared memory.
// Follows the reference's sequence: f32 maximum, exp((f64)(v - max)) with the subtraction in f32,
// the f64 sum accumulated in ascending expert order by one lane, f32 weights, then k rounds of
// "largest weight, lowest index" and a renormalisation summed in ascending index order.
template <int EPL>
__device__ __forceinline__ int route_one_warp(const float* lg, int E, int k, int renormalize, int lane,
                                              int32_t* idx_out, float* w_out, double* exps /* smem, E */) {
  float mx = -INFINITY;
  bool finite = true;
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    int e = lane + 32 * j;
    if (e < E) {
      float v = lg[e];
      if (!isfinite(v)) finite = false;
      mx = fmaxf(mx, v);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (__any_sync(0xffffffffu, !finite)) return ATENIA_ERR_ROUTING;
  double ex[EPL];
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    int e = lane + 32 * j;
    ex[j] = 0.0;
    if (e < E) {
      ex[j] = exp((double)__fsub_rn(lg[e], mx));
      exps[e] = ex[j];
    }
  }
  __syncwarp();
  double sum = 0.0;
  if (lane == 0)
    for (int e = 0; e < E; ++e) sum += exps[e];
  sum = __shfl_sync(0xffffffffu, sum, 0);
  const double inv = sum > 0.0 ? 1.0 / sum : 0.0;
  float p[EPL];
  bool taken[EPL];
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    p[j] = (float)(ex[j] * inv);
    taken[j] = (lane + 32 * j) >= E;  // slots past E never compete
  }
  for (int s = 0; s < k; ++s) {
    float bw = -1.0f;  // weights are >= 0
    int bi = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      if (!taken[j] && p[j] > bw) {  // ascending j = ascending index: strict > keeps the lower one
        bw = p[j];
        bi = lane + 32 * j;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ow = __shfl_xor_sync(0xffffffffu, bw, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ow > bw || (ow == bw && oi < bi)) {
        bw = ow;
        bi = oi;
      }
    }
#pragma unroll
    for (int j = 0; j < EPL; ++j)
      if (lane + 32 * j == bi) taken[j] = true;
  }
  // selected experts in ascending order: rank of each selected slot among the selected
  int m_before = 0;
  double ssum = 0.0;
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    bool sel = taken[j] && (lane + 32 * j) < E;
    unsigned mask = __ballot_sync(0xffffffffu, sel);
    int rank = m_before + __popc(mask & ((1u << lane) - 1u));
    if (sel) {
      idx_out[rank] = lane + 32 * j;
      exps[rank] = (double)p[j];  // reuse as the selected-weight list (ascending index)
    }
    m_before += __popc(mask);
  }
  __syncwarp();
  if (lane == 0)
    for (int s = 0; s < k; ++s) ssum += exps[s];
  ssum = __shfl_sync(0xffffffffu, ssum, 0);
  if (!(ssum > 0.0)) return ATENIA_ERR_ROUTING;
  const double scale = renormalize ? 1.0 / ssum : 1.0;
  if (lane < k) w_out[lane] = (float)(exps[lane] * scale);
  __syncwarp();
  return 0;
}

// The same for NT tokens by one warp at a time: what one token leaves idle (the serial sum runs in one lane, every step
// waits for a shuffle) the others fill.  Token j has its logits at lg + j * lg_ld and its scratch at exps + j * exps_ld
// (exps_ld odd: lane j adds token j's values); rc[j] as route_one_warp returns it, for tokens that are `valid`.
template <int EPL, int NT>
__device__ __forceinline__ void route_many_warp(const float* lg, int lg_ld, const bool (&valid)[NT], int E, int k,
                                                int renormalize, int lane, int32_t (*idx_out)[kMaxK],
                                                float (*w_out)[kMaxK], double* exps, int exps_ld, int (&rc)[NT]) {
  double inv[NT];
  float p[NT][EPL];
  bool taken[NT][EPL];
  {
    double ex[NT][EPL];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      rc[t] = 0;
      float v[EPL], mx = -INFINITY;
      bool finite = true;
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        v[j] = valid[t] && e < E ? lg[t * lg_ld + e] : -INFINITY;
        if (valid[t] && e < E && !isfinite(v[j])) finite = false;
        mx = fmaxf(mx, v[j]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (__any_sync(0xffffffffu, !finite)) rc[t] = ATENIA_ERR_ROUTING;
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        ex[t][j] = 0.0;
        if (valid[t] && e < E) {
          ex[t][j] = exp((double)__fsub_rn(v[j], mx));
          exps[t * exps_ld + e] = ex[t][j];
        }
      }
    }
    __syncwarp();
    double sum = 0.0;
    if (lane < NT)
      for (int e = 0; e < E; ++e) sum += exps[lane * exps_ld + e];
    const double mine = sum > 0.0 ? 1.0 / sum : 0.0;
    __syncwarp();
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      inv[t] = __shfl_sync(0xffffffffu, mine, t);
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        p[t][j] = (float)(ex[t][j] * inv[t]);
        taken[t][j] = (lane + 32 * j) >= E;
      }
    }
  }
  for (int s = 0; s < k; ++s) {
    float bw[NT];
    int bi[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      bw[t] = -1.0f;
      bi[t] = 0x7fffffff;
#pragma unroll
      for (int j = 0; j < EPL; ++j)
        if (!taken[t][j] && p[t][j] > bw[t]) {
          bw[t] = p[t][j];
          bi[t] = lane + 32 * j;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const float ow = __shfl_xor_sync(0xffffffffu, bw[t], o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi[t], o);
        if (ow > bw[t] || (ow == bw[t] && oi < bi[t])) {
          bw[t] = ow;
          bi[t] = oi;
        }
      }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j = 0; j < EPL; ++j)
        if (lane + 32 * j == bi[t]) taken[t][j] = true;
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    int m_before = 0;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      const bool sel = valid[t] && rc[t] == 0 && taken[t][j] && (lane + 32 * j) < E;
      const unsigned mask = __ballot_sync(0xffffffffu, sel);
      const int rank = m_before + __popc(mask & ((1u << lane) - 1u));
      if (sel && rank < kMaxK) {
        idx_out[t][rank] = lane + 32 * j;
        exps[t * exps_ld + rank] = (double)p[t][j];  // reuse as the selected-weight list (ascending index)
      }
      m_before += __popc(mask);
    }
  }
  __syncwarp();
  double ssum = 0.0;
  if (lane < NT)
    for (int s = 0; s < k; ++s) ssum += exps[lane * exps_ld + s];
  const double mine = renormalize ? 1.0 / ssum : 1.0;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const double total = __shfl_sync(0xffffffffu, ssum, t), scale = __shfl_sync(0xffffffffu, mine, t);
    if (!(total > 0.0)) rc[t] = ATENIA_ERR_ROUTING;
    if (lane < k) w_out[t][lane] = (float)(exps[t * exps_ld + lane] * scale);
  }
  __syncwarp();
}

}  // namespace atenia
