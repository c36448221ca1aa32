// Dispatch: the canonical permutation of (token, slot) entries by expert, and the row gather.
//
// The reference never builds a permutation: it loops over tokens in order and, inside a token, over
// the selected experts in ascending order (src/moe/graph_op.rs:346-348, src/moe/sparse.rs:173-175).
// The only order it defines is therefore "tokens ascending, experts ascending inside a token", and
// the permutation emitted here is the stable counting sort of the flat entry list i = t*k + s by
// expert id: expert_offsets[e] = number of entries with a smaller expert, and the rows of one
// expert keep ascending i.  Three launches (per-block histogram, scan, stable placement) above 16384
// entries, one below.
#include "common.cuh"

namespace atenia {
namespace {

constexpr int kMaxE = 128;

__global__ void __launch_bounds__(kDispatchChunk) count_kernel(DispatchArgs a) {
  __shared__ int hist[kMaxE];
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  int i = blockIdx.x * kDispatchChunk + threadIdx.x;
  if (i < a.n) {
    int e = a.topk_idx[i];
    if (e < 0 || e >= a.E) {
      report_error(a.err, ATENIA_ERR_ROUTING, 2000);
    } else {
      atomicAdd(&hist[e], 1);
    }
  }
  __syncthreads();
  // counts are kept expert-major, [E][gridDim.x]: the scan then reads consecutive blocks of one expert
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) a.block_counts[(size_t)e * gridDim.x + blockIdx.x] = hist[e];
}

// One block.  Warp w scans experts w, w + nwarps, ... over the blocks (32 blocks per step, the loads of
// up to eight steps issued before the first is consumed); then thread 0 scans experts.
__global__ void __launch_bounds__(1024) scan_kernel(DispatchArgs a, int nblk) {
  __shared__ int totals[kMaxE];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  constexpr int kBatch = 8;
  for (int e = warp; e < a.E; e += nwarps) {
    const int32_t* cnt = a.block_counts + (size_t)e * nblk;
    int32_t* base = a.block_base + (size_t)e * nblk;
    int running = 0;
    for (int b0 = 0; b0 < nblk; b0 += 32 * kBatch) {
      int c[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int b = b0 + 32 * j + lane;
        c[j] = b < nblk ? cnt[b] : 0;
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int b = b0 + 32 * j + lane;
        int incl = c[j];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (b < nblk) base[b] = running + incl - c[j];
        running += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    if (lane == 0) totals[e] = running;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int e = 0; e < a.E; ++e) {
      a.expert_offsets[e] = run;
      run += totals[e];
    }
    a.expert_offsets[a.E] = run;
    if (a.extra_offsets) {
      a.extra_offsets[0] = 0;
      a.extra_offsets[1] = a.T;
    }
  }
}

__global__ void __launch_bounds__(kDispatchChunk) place_kernel(DispatchArgs a) {
  constexpr int kW = kDispatchChunk / 32;
  __shared__ int warp_cnt[kW][kMaxE];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j = threadIdx.x; j < kW * kMaxE; j += blockDim.x) (&warp_cnt[0][0])[j] = 0;
  __syncthreads();
  const int i = blockIdx.x * kDispatchChunk + threadIdx.x;
  int e = -1;
  if (i < a.n) {
    e = a.topk_idx[i];
    if (e < 0 || e >= a.E) e = -1;
  }
  // lanes holding the same expert, in lane order = entry order
  const unsigned peers = __match_any_sync(0xffffffffu, e);
  const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
  if (e >= 0 && rank_in_warp == 0) warp_cnt[warp][e] = __popc(peers);
  __syncthreads();
  if (e >= 0) {
    int before = 0;
    for (int w = 0; w < warp; ++w) before += warp_cnt[w][e];
    const int pos = a.expert_offsets[e] + a.block_base[(size_t)e * gridDim.x + blockIdx.x] + before + rank_in_warp;
    a.perm[pos] = i;
    a.inv_perm[i] = pos;
  } else if (i < a.n) {
    a.inv_perm[i] = -1;  // an entry with an invalid expert id has no row: the combine skips it
  }
}

// Small batches (at most 1024 entries, i.e. decode): histogram, scan and stable placement in ONE block,
// one thread per entry -- the same permutation as the three launches above without their launch gaps.
constexpr int kSmallDispatchMax = 1024;

__global__ void __launch_bounds__(kSmallDispatchMax) dispatch_small_kernel(DispatchArgs a) {
  __shared__ int warp_cnt[kSmallDispatchMax / 32][kMaxE];  // entries of expert e in warp w, then their base
  __shared__ int offsets[kMaxE + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  chain_next();
  for (int j = threadIdx.x; j < nwarps * kMaxE; j += blockDim.x) (&warp_cnt[0][0])[j] = 0;
  chain_wait();
  __syncthreads();
  const int i = threadIdx.x;
  int e = -1;
  if (i < a.n) {
    e = a.topk_idx[i];
    if (e < 0 || e >= a.E) {
      report_error(a.err, ATENIA_ERR_ROUTING, 2001);
      e = -1;
    }
  }
  const unsigned peers = __match_any_sync(0xffffffffu, e);
  const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
  if (e >= 0 && rank_in_warp == 0) warp_cnt[warp][e] = __popc(peers);
  __syncthreads();
  // thread e: exclusive scan of its expert's counts over the warps (entry order), total into offsets
  if (threadIdx.x < a.E) {
    int run = 0;
    for (int w = 0; w < nwarps; ++w) {
      const int c = warp_cnt[w][threadIdx.x];
      warp_cnt[w][threadIdx.x] = run;
      run += c;
    }
    offsets[threadIdx.x + 1] = run;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    offsets[0] = 0;
    for (int x = 0; x < a.E; ++x) offsets[x + 1] += offsets[x];
    if (a.extra_offsets) {
      a.extra_offsets[0] = 0;
      a.extra_offsets[1] = a.T;
    }
  }
  __syncthreads();
  for (int x = threadIdx.x; x <= a.E; x += blockDim.x) a.expert_offsets[x] = offsets[x];
  if (e >= 0) {
    const int pos = offsets[e] + warp_cnt[warp][e] + rank_in_warp;
    a.perm[pos] = i;
    a.inv_perm[i] = pos;
  } else if (i < a.n) {
    a.inv_perm[i] = -1;
  }
}

// Medium batches (at most 16384 entries): the same in ONE launch of one cluster of eight CTAs, each with an eighth
// of the entries: histogram (shared-memory atomics; the order of additions does not matter for counts), the
// eight histograms read through distributed shared memory, then per chunk of 1024 entries the stable placement
// of dispatch_small_kernel, the warps' counts scanned by one warp per expert.  Latency, not bandwidth, is what
// it takes: Mixtral shape, 4096 tokens, 14.8 us in one block, 4.7 in the cluster.  Larger batches keep the three
// launches: with 49152 entries beside a shared expert's GEMM 22 us against 34 (six chunks per CTA in turn).
constexpr int kClusterDispatchMax = 16384;
constexpr int kDispatchCtas = 8;

__global__ void __cluster_dims__(kDispatchCtas, 1, 1) __launch_bounds__(kSmallDispatchMax)
dispatch_cluster_kernel(DispatchArgs a) {
  constexpr int kWarps = kSmallDispatchMax / 32;
  // entries of expert e in warp w of the chunk, then those of the warps before it.  16 bits: with 32 the block's 18 KB
  // would not fit beside a CTA of the expert GEMMs, which is where a shared expert's run at that time.
  __shared__ uint16_t warp_cnt[kWarps][kMaxE + 2];  // (row length: 65 words, the scan reads a column)
  __shared__ int hist[kMaxE];     // entries per expert of this CTA
  __shared__ int totals[kMaxE];   // ... of all CTAs
  __shared__ int next_row[kMaxE]; // next row of each expert for this CTA's entries
  __shared__ int chunk_row[kMaxE];  // ... as the current chunk began
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x;  // the grid is one cluster
  const int per = ((a.n + kDispatchCtas - 1) / kDispatchCtas + 31) & ~31;
  const int begin = rank * per < a.n ? rank * per : a.n;
  const int end = begin + per < a.n ? begin + per : a.n;
  chain_next();
  if (threadIdx.x < kMaxE) hist[threadIdx.x] = 0;
  chain_wait();
  __syncthreads();
  for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
    const int e = a.topk_idx[i];
    if (e >= 0 && e < a.E) atomicAdd(&hist[e], 1);
    else report_error(a.err, ATENIA_ERR_ROUTING, 2002);
  }
  __syncwarp();  // (.aligned: the lanes of a warp arrive together, and the loop lets them leave apart)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  int before = 0, total = 0;
  if (threadIdx.x < a.E) {
    const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(&hist[threadIdx.x]));
#pragma unroll
    for (int r = 0; r < kDispatchCtas; ++r) {
      uint32_t theirs;
      int c;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(r));
      asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(c) : "r"(theirs) : "memory");
      if (r < rank) before += c;
      total += c;
    }
    totals[threadIdx.x] = total;
  }
  // (waited for at the end: no CTA leaves while another may read its histogram)
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the totals, four experts per lane
    int c[kMaxE / 32], sum = 0;
#pragma unroll
    for (int j = 0; j < kMaxE / 32; ++j) {
      const int e = lane * (kMaxE / 32) + j;
      c[j] = e < a.E ? totals[e] : 0;
      sum += c[j];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    int run = incl - sum;
#pragma unroll
    for (int j = 0; j < kMaxE / 32; ++j) {
      const int e = lane * (kMaxE / 32) + j;
      if (e < a.E) {
        totals[e] = run;
        if (rank == 0) a.expert_offsets[e] = run;
      }
      run += c[j];
    }
    if (rank == 0 && lane == 31) {
      a.expert_offsets[a.E] = run;
      if (a.extra_offsets) {
        a.extra_offsets[0] = 0;
        a.extra_offsets[1] = a.T;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < a.E) next_row[threadIdx.x] = totals[threadIdx.x] + before;
  for (int c0 = begin; c0 < end; c0 += kSmallDispatchMax) {
    for (int e = lane; e < a.E; e += 32) warp_cnt[warp][e] = 0;
    __syncwarp();
    const int i = c0 + threadIdx.x;
    int e = -1;
    if (i < end) {
      e = a.topk_idx[i];
      if (e < 0 || e >= a.E) e = -1;  // (reported by the histogram pass)
    }
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
    if (e >= 0 && rank_in_warp == 0) warp_cnt[warp][e] = (uint16_t)__popc(peers);
    __syncthreads();
    for (int x = warp; x < a.E; x += kWarps) {
      const int c = warp_cnt[lane][x];
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      warp_cnt[lane][x] = (uint16_t)(incl - c);
      if (lane == 31) {
        const int row = next_row[x];
        chunk_row[x] = row;
        next_row[x] = row + incl;
      }
    }
    __syncthreads();
    if (e >= 0) {
      const int pos = chunk_row[e] + warp_cnt[warp][e] + rank_in_warp;
      a.perm[pos] = i;
      a.inv_perm[i] = pos;
    } else if (i < end) {
      a.inv_perm[i] = -1;
    }
    __syncwarp();  // (a warp's row is cleared by the warp itself)
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Row gather: x_perm[r, :] = bf16(x[perm[r] / k, :]).  One warp per destination row, eight rows per
// block in flight and a grid that loops; every lane keeps four 16-byte vectors in flight.  `placed`
// points at expert_offsets[E], the number of rows the placement actually wrote: entries with an
// invalid expert id get no row, so perm beyond that count holds whatever an earlier call left there
// and must not be followed.  Rows n_rows .. n_rows + T - 1 of the index space convert x itself
// (f32 input with a shared expert: x_bf16 = bf16(x)).
constexpr int kGatherWarps = 8;

__global__ void __launch_bounds__(kGatherWarps * 32) gather_rows_kernel(const void* __restrict__ x, int x_is_f32,
                                                                         const int32_t* __restrict__ perm,
                                                                         const int32_t* __restrict__ placed,
                                                                         int n_rows, int k, int d,
                                                                         __nv_bfloat16* __restrict__ x_perm,
                                                                         __nv_bfloat16* __restrict__ x_bf16, int T,
                                                                         int total_rows) {
  const int lane = threadIdx.x & 31;
  const int nvec = d / 8;
  chain_wait();
  chain_next();  // (after the wait: the GEMM behind takes every SM, so it may come no earlier than these rows)
  const int n_placed = n_rows > 0 ? *placed : 0;
  for (int r = blockIdx.x * kGatherWarps + (threadIdx.x >> 5); r < total_rows; r += gridDim.x * kGatherWarps) {
    int src_t, dst_r;
    __nv_bfloat16* dst;
    if (r < n_rows) {
      if (r >= n_placed) continue;
      src_t = perm[r] / k;
      if (src_t < 0 || src_t >= T) continue;
      dst_r = r;
      dst = x_perm;
    } else {
      src_t = r - n_rows;
      dst_r = src_t;
      dst = x_bf16;
    }
    uint4* drow = reinterpret_cast<uint4*>(dst + (size_t)dst_r * d);
    if (x_is_f32) {
      const float4* srow = reinterpret_cast<const float4*>(static_cast<const float*>(x) + (size_t)src_t * d);
      for (int v = lane; v < nvec; v += 64) {
        float4 a0 = srow[2 * v], b0 = srow[2 * v + 1], a1, b1;
        const bool two = v + 32 < nvec;
        if (two) {
          a1 = srow[2 * (v + 32)];
          b1 = srow[2 * (v + 32) + 1];
        }
        drow[v] = make_uint4(pack_bf16x2(a0.x, a0.y), pack_bf16x2(a0.z, a0.w), pack_bf16x2(b0.x, b0.y),
                             pack_bf16x2(b0.z, b0.w));
        if (two)
          drow[v + 32] = make_uint4(pack_bf16x2(a1.x, a1.y), pack_bf16x2(a1.z, a1.w), pack_bf16x2(b1.x, b1.y),
                                    pack_bf16x2(b1.z, b1.w));
      }
    } else {
      const uint4* srow = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(x) + (size_t)src_t * d);
      for (int v = lane; v < nvec; v += 128) {
        uint4 t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (v + 32 * j < nvec) t[j] = srow[v + 32 * j];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (v + 32 * j < nvec) drow[v + 32 * j] = t[j];
      }
    }
  }
}

}  // namespace

int launch_dispatch(const DispatchArgs& a, cudaStream_t s) {
  if (a.E > kMaxE) return ATENIA_ERR_UNSUPPORTED;
  if (a.n > 0 && a.n <= kSmallDispatchMax) {
    const int threads = ((a.n + 31) / 32 * 32) < a.E ? ((a.E + 31) / 32 * 32) : ((a.n + 31) / 32 * 32);
    count_launch();
    return launch_chained(a.chained, dispatch_small_kernel, dim3(1), dim3(threads), 0, s, a);
  }
  if (a.n > kSmallDispatchMax && a.n <= kClusterDispatchMax) {
    count_launch();
    return launch_chained(a.chained, dispatch_cluster_kernel, dim3(kDispatchCtas), dim3(kSmallDispatchMax), 0, s, a);
  }
  const int nblk = (a.n + kDispatchChunk - 1) / kDispatchChunk;
  if (nblk > 0) {
    count_kernel<<<nblk, kDispatchChunk, 0, s>>>(a);
    count_launch();
  }
  scan_kernel<<<1, 1024, 0, s>>>(a, nblk);
  count_launch();
  if (nblk > 0) {
    place_kernel<<<nblk, kDispatchChunk, 0, s>>>(a);
    count_launch();
  }
  return (int)cudaGetLastError();
}

int launch_gather_rows(const void* x, int x_is_f32, const int32_t* perm, const int32_t* placed, int n_rows, int k,
                       int d, __nv_bfloat16* x_perm, __nv_bfloat16* x_bf16, int T, bool chained, cudaStream_t s) {
  const int extra = x_bf16 ? T : 0;
  const int total = n_rows + extra;
  if (total <= 0) return ATENIA_OK;
  // enough blocks to keep every SM's memory pipeline full; the kernel loops over the rest
  const int want = (total + kGatherWarps - 1) / kGatherWarps;
  const int cap = 148 * 8;
  count_launch();
  return launch_chained(chained, gather_rows_kernel, dim3(want < cap ? want : cap), dim3(kGatherWarps * 32), 0, s, x, x_is_f32, perm,
                        placed, n_rows, k, d, x_perm, x_bf16, T, total);
}

}  // namespace atenia
