// Grouped expert GEMM for bf16 weights with CTA pairs (tcgen05 cta_group::2), transposed: the weights are
// the M side, the token rows the N side of the MMA.
//
// Two CTAs on the two SMs of a TPC form a cluster and compute D[f, t] = sum_k W[f, k] X[t, k] for 256 weight
// rows (128 in each CTA's tensor memory) and a token tile of n <= 256 rows, n a multiple of 16.  Each CTA
// stages its own 128 weight rows and half of the token tile; one thread of the leader CTA issues
// tcgen05.mma.cta_group::2 (M256 x Nn x K16), which reads both operands from both CTAs' shared memory.
//
// Why transposed: the M side of an MMA costs 256 rows however few hold data, the N side costs what it is
// wide.  A group of R rows is cut into ceil(R / 256) (192, 128, 64) equal token tiles rounded up to 16 rows, so the padding
// is below 16 rows per tile.
//
//   kSwiGLU : 256 weight rows = 128 features; a CTA's 128 rows are 64 rows of W_gate and the same 64 of W_up,
//             so the epilogue warps of lane quarters q and q + 2 hold gate and up of the same features and
//             exchange them through shared memory (f32), each finishing half of the tokens
//   kPlain  : 256 weight rows = 256 features
//   k-block : 64 (one 128-byte swizzle row): 16 KiB of weights + 16, 12, 8 or 4 KiB of tokens per CTA (tiles of at most 256,
//             192, 128 or 64 token rows, the launch's choice: pair_tokens_of), 6, 7, 8 or 10 stages
//
// What bounds it: below some hundred rows per group HBM's latency, that is, the weights in flight (10 stages hold 160 KiB per
// SM: 16 tokens of the Mixtral shape 451 -> 422 us against 6 stages), above the tensor pipe and the board's power.  ncu, DeepSeek-V2-Lite shape, 8192 tokens, gate/up: the
// pipe is busy 90 % of 524 k cycles (75 % of 626 k with the issuing lane under `lane == 0`, see uniform_warp;
// 67 % of 701 k with two token tiles per weight tile and 16-byte stores through shared memory).  One forward on a
// B200, before (token-major 256-row pair tiles from 512 rows per group, 128-row single-CTA tiles below) and now:
// Mixtral shape 256 / 4096 tokens 548 -> 514 / 2710 -> 2605 us (power-capped), Qwen1.5-MoE shape 2048 tokens
// 453 -> 410, DeepSeek-V2-Lite shape 61 / 8192 tokens 284 -> 263 / 1259 -> 1193, a 512-wide layer of 64 tokens
// 53.6 -> 50.1.
// No TMA multicast is used: every CTA fetches its own tiles (cp.async.bulk.tensor ... cta_group::2
// only routes the completion to the leader's mbarrier).
//
// Barriers: full[s] lives in the leader and collects the bytes of both CTAs; empty[s] and
// acc_full[b] exist in both CTAs and are signalled by tcgen05.commit with a CTA mask; acc_empty[b]
// lives in the leader and is arrived on by the epilogue warps of both CTAs.
#include <type_traits>

#include "tc_common.cuh"

namespace atenia {
namespace {
using namespace tc;

constexpr int TN2 = kPairTokens;
constexpr int MAX_STAGES2 = 10;
constexpr int ACC_BUFS2 = 2;
constexpr int TMEM_COLS2 = 512;
constexpr int W_BYTES2 = BM * BK * 2;         // 16 KiB: this CTA's 128 weight rows
constexpr int EPI_WARPS2 = 8;
constexpr int NUM_THREADS2 = 64 + EPI_WARPS2 * 32;
constexpr int EPI_WARP_BYTES2 = 2 * 1024;  // kSwiGLU: two buffers of 8 tokens x 32 features of f32 per warp
constexpr int EPI_BYTES2 = EPI_WARPS2 * EPI_WARP_BYTES2;
// The ring by the token rows of a tile at most.
template <int TOK>
struct PairRing {
  static constexpr int X_BYTES = (TOK / 2) * BK * 2;  // this CTA's half of the token tile
  static constexpr int STAGE_BYTES = W_BYTES2 + X_BYTES;
  static constexpr int STAGES = TOK == 256 ? 6 : TOK == 192 ? 7 : TOK == 128 ? 8 : 10;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES2 + 1024 + 256;
  static_assert(STAGES <= MAX_STAGES2 && STAGE_BYTES % 1024 == 0 && SMEM_BYTES <= 225 * 1024, "");
};

struct __align__(8) Barriers2 {
  uint64_t full[MAX_STAGES2];
  uint64_t empty[MAX_STAGES2];
  uint64_t acc_full[ACC_BUFS2];
  uint64_t acc_empty[ACC_BUFS2];
  uint32_t tmem_base;
  int abort_flag;
};

// D f32, A = B = bf16, K-major, M = 256 (per pair); N is added per tile.
constexpr uint32_t kInstrDesc2 = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(256 >> 4) << 24);

// ---- tile walk: the token tiles of one group are equal, so none is a nearly empty remainder ----
struct PairCursor {
  int group, base;  // current group, first tile index of it
  int m_tiles, tile_rows;
  int row_begin, row_end;
};
struct PairTile {
  int group, row0, rows, f0;  // first row and rows of the tile, first feature
  int n;                      // MMA N: rows rounded up to 16
};
template <int TOK>
__device__ __forceinline__ void pair_cursor_load(PairCursor& c, const int32_t* __restrict__ off) {
  c.row_begin = off[c.group];
  c.row_end = off[c.group + 1];
  const int rows = c.row_end - c.row_begin;
  c.m_tiles = pair_tiles(rows, TOK);
  c.tile_rows = pair_tile_rows(rows, c.m_tiles);
}
template <int TOK>
__device__ __forceinline__ bool pair_cursor_seek(PairCursor& c, int tile, int f_tiles, int num_groups,
                                                 const int32_t* __restrict__ off, PairTile& out, int f_width) {
  while (c.group < num_groups) {
    const int here = c.m_tiles * f_tiles;
    if (tile < c.base + here) {
      const int local = tile - c.base;
      const int ft = local / c.m_tiles;  // token tiles of one weight tile are neighbours: they share it in L2
      const int mt = local - ft * c.m_tiles;
      out.group = c.group;
      out.row0 = c.row_begin + mt * c.tile_rows;
      out.rows = min(c.row_end - out.row0, c.tile_rows);  // >= 1: m_tiles is the fewest of tile_rows
      out.n = pair_tile_n(out.rows);
      out.f0 = ft * f_width;
      return true;
    }
    c.base += here;
    c.group += 1;
    if (c.group < num_groups) pair_cursor_load<TOK>(c, off);
  }
  return false;
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `addr` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The following run in a converged warp; one lane (always the same) issues the instruction.
// TMA load whose completion bytes go to an mbarrier that may live in the peer CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int x,
                                                 int y) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(x), "r"(y)
      : "memory");
}
// The four MMAs (K = 16 each, 32 bytes apart inside the swizzle row) of one k-block.
__device__ __forceinline__ void tc_mma_bf16_pair_kblock(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                                        uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred e, p, t;\n\t"
      ".reg .b64 a, b;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "add.s64 a, %1, 2;\n\tadd.s64 b, %2, 2;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 4;\n\tadd.s64 b, %2, 4;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 6;\n\tadd.s64 b, %2, 6;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, t;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive (once the MMAs issued so far have completed) on the barrier at this offset in both CTAs.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
      ::"r"(bar), "h"(mask)
      : "memory");
}

// One more group in the launch (GroupedGemmArgs::Extra): its tiles come first.
struct PairExtra {
  PairRowMaps x;
  const CUtensorMap* w0;
  const CUtensorMap* w1;
  __nv_bfloat16* out;
  int rows, N, K;
};
struct NoExtra {};

template <int MODE, int TOK, bool EX>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS2, 1)
grouped_gemm_2cta_kernel(const __grid_constant__ PairRowMaps tmaps_x, const CUtensorMap* __restrict__ tmap_w0,
                         const CUtensorMap* __restrict__ tmap_w1, const int32_t* __restrict__ group_offsets_g,
                         int num_groups, int N, int K, __nv_bfloat16* __restrict__ out, DeviceError* err,
                         const __grid_constant__ std::conditional_t<EX, PairExtra, NoExtra> ex) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int32_t goff_s[kMaxGroupsShared + 1];
  constexpr int F_CTA = (MODE == kSwiGLU) ? BM / 2 : BM;  // output features per CTA
  constexpr int F_PAIR = 2 * F_CTA;
  constexpr int STAGES2 = PairRing<TOK>::STAGES, STAGE_BYTES2 = PairRing<TOK>::STAGE_BYTES;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_aligned = smem_raw + (smem_base - smem_u32(smem_raw));
  uint8_t* epi = smem_aligned + STAGES2 * STAGE_BYTES2;
  Barriers2* bars = reinterpret_cast<Barriers2*>(epi + EPI_BYTES2);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = uniform_warp();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int num_kb = (K + BK - 1) / BK;
  const int f_tiles = (N + F_PAIR - 1) / F_PAIR;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) {
      mbar_init(smem_u32(&bars->full[s]), 1);
      mbar_init(smem_u32(&bars->empty[s]), 1);
    }
    for (int b = 0; b < ACC_BUFS2; ++b) {
      mbar_init(smem_u32(&bars->acc_full[b]), 1);
      mbar_init(smem_u32(&bars->acc_empty[b]), 2 * EPI_WARPS2);  // the epilogue warps of both CTAs
    }
    bars->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&bars->tmem_base)),
                 "r"(TMEM_COLS2)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  // before chain_wait(): the group offsets and, below, the first weights (see chain_wait)
  stage_group_offsets(group_offsets_g, num_groups, goff_s);
  const int32_t* group_offsets = goff_s;
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // barriers of both CTAs are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  PairCursor cur;
  cur.group = 0;
  cur.base = 0;
  if (num_groups > 0) pair_cursor_load<TOK>(cur, group_offsets);
  PairTile tc;
  int ex_m = 1, ex_rows = 16, ex_kb = 0;
  PairDeal deal{};
  if constexpr (EX) {
    ex_m = pair_tiles(ex.rows, TOK);
    ex_rows = pair_tile_rows(ex.rows, ex_m);
    ex_kb = (ex.K + BK - 1) / BK;
    deal = pair_deal(num_pairs, ex_m * ((ex.N + F_PAIR - 1) / F_PAIR), ex_kb, num_kb);
  }
  // This pair's i-th tile (the extra group is group -1); false past its last.
  auto seek = [&](PairCursor& c, int i) {
    int tile = pair + i * num_pairs;
    if constexpr (EX) {
      bool extra;
      tile = pair_deal_tile(deal, pair, i, extra);
      if (extra) {
        const int ft = tile / ex_m, mt = tile - ft * ex_m;
        tc.group = -1;
        tc.row0 = mt * ex_rows;
        tc.rows = min(ex.rows - tc.row0, ex_rows);
        tc.n = pair_tile_n(tc.rows);
        tc.f0 = ft * F_PAIR;
        return true;
      }
    }
    return pair_cursor_seek<TOK>(c, tile, f_tiles, num_groups, group_offsets, tc, F_PAIR);
  };
  auto k_blocks = [&] { return EX && tc.group < 0 ? ex_kb : num_kb; };
  auto weights0 = [&] {
    if constexpr (EX) return tc.group < 0 ? ex.w0 : &tmap_w0[tc.group];
    else return &tmap_w0[tc.group];
  };
  auto weights1 = [&] {
    if constexpr (EX) return tc.group < 0 ? ex.w1 : &tmap_w1[tc.group];
    else return &tmap_w1[tc.group];
  };

  if (warp == 0) {
    // ================= TMA producer (both CTAs) =================
    int stage = 0;
    uint32_t phase = 0;
    int last_group = -2;
    uint32_t armed = 0;  // stages with a copy possibly in flight
    bool ok = true;
    // Weights of the first tile's first k-blocks; their token rows follow after the wait.  B200, 64 tokens of a 512-wide
    // layer 37.7 -> 33.9 us, 256 Mixtral tokens 507 -> 497.
    int ahead = 0;
    // (The loop's first seek finds the cursor where this one left it.  Walking the groups again there delays the token rows: 32
    // experts of 512 x 1408, shared 2816 on the second stream, 333 / 500 / 1000 tokens 70.8 / 73.5 / 89.7 -> 67.2 / 70.5 / 86.1 us a
    // forward.  In streams of weights, tiles of 64 rows or an extra group, the CTAs had better not start as one, and the walk is
    // repeated: once / twice 64 top-2 experts of 2048 x 1408 and a shared one, 24 tokens 112.1 / 111.2, 128 top-2 of 2048 x 768 and a
    // shared one, 24 / 100 tokens 96.0 / 93.9, 171.6 / 170.1; alone, 96 top-8 of 3072 x 1024, 3 tokens 99.7 / 96.6, 64 top-1 of 4096 x 512, 28
    // tokens 88.5 / 86.6, 128 top-1 of 4096 x 1024, 31 tokens 155.3 / 152.4.)
    PairCursor first = cur;
    const bool any = seek(first, 0);
    if constexpr (!EX && TOK > 64) cur = first;
    if (any) {
      const CUtensorMap* m0 = weights0();
      const CUtensorMap* m1 = MODE == kSwiGLU ? weights1() : m0;
      tmap_acquire(m0);
      if (MODE == kSwiGLU) tmap_acquire(m1);
      last_group = tc.group;
      const int nkb = k_blocks();
      ahead = nkb < STAGES2 ? nkb : STAGES2;
      const uint32_t tx = 2 * (W_BYTES2 + pair_box_rows(pair_tile_box(tc.n)) * BK * 2);
      const int f_row = tc.f0 + (int)rank * F_CTA;
      for (int kb = 0; kb < ahead; ++kb) {
        const uint32_t full_local = smem_u32(&bars->full[kb]);
        const uint32_t full_leader = mapa(full_local, 0);
        const uint32_t dst = smem_base + kb * STAGE_BYTES2;
        if (leader) mbar_expect_tx_one(full_local, tx);
        tma_load_2d_pair(dst, m0, full_leader, kb * BK, f_row);
        if (MODE == kSwiGLU) tma_load_2d_pair(dst + W_BYTES2 / 2, m1, full_leader, kb * BK, f_row);
      }
    }
    chain_wait();
    for (int i = 0; ok && seek(cur, i); ++i) {
      const CUtensorMap* m0 = weights0();
      const CUtensorMap* m1 = MODE == kSwiGLU ? weights1() : m0;
      if (tc.group != last_group) {
        tmap_acquire(m0);
        if (MODE == kSwiGLU) tmap_acquire(m1);
        last_group = tc.group;
      }
      const int box = pair_tile_box(tc.n);
      const CUtensorMap* mx = &tmaps_x.box[box];
      if constexpr (EX) {
        if (tc.group < 0) mx = &ex.x.box[box];
      }
      const int nkb = k_blocks();
      const int f_row = tc.f0 + (int)rank * F_CTA;
      const int x_row = tc.row0 + (int)rank * (tc.n / 2);
      const uint32_t tx = 2 * (W_BYTES2 + pair_box_rows(box) * BK * 2);  // bytes of both CTAs
      for (int kb = 0; kb < nkb; ++kb) {
        const uint32_t full_local = smem_u32(&bars->full[stage]);
        const uint32_t full_leader = mapa(full_local, 0);
        const uint32_t dst = smem_base + stage * STAGE_BYTES2;
        if (ahead > 0) {  // (the first tile: its weights are on their way)
          --ahead;
        } else {
          if (!mbar_wait(smem_u32(&bars->empty[stage]), phase ^ 1u, abort_flag)) {
            if (lane == 0) report_error(err, ATENIA_ERR_DEVICE_TIMEOUT, 1100 + stage);
            *abort_flag = 1;
            ok = false;
          }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (leader) mbar_expect_tx_one(full_local, tx);
          tma_load_2d_pair(dst, m0, full_leader, kb * BK, f_row);
          if (MODE == kSwiGLU) tma_load_2d_pair(dst + W_BYTES2 / 2, m1, full_leader, kb * BK, f_row);
        }
        tma_load_2d_pair(dst + W_BYTES2, mx, full_leader, kb * BK, x_row);
        armed |= 1u << stage;
        if (++stage == STAGES2) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    chain_next();  // (every load is on its way: what follows may be launched)
    if (*abort_flag && leader && lane == 0) {
      // let the copies already issued (both CTAs') land before the pair's shared memory is released
      for (int s = 0; s < STAGES2; ++s) {
        if (!(armed & (1u << s))) continue;
        const uint32_t par = s < stage ? phase : phase ^ 1u;
        for (int i = 0; i < (1 << 16) && !mbar_try_wait(smem_u32(&bars->full[s]), par); ++i) {}
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (leader CTA only) =================
    chain_wait();
    if (leader) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase = 0;  // bit b: accumulator b
      int it = 0;
      bool ok = true;
      for (; ok && seek(cur, it); ++it) {
        const int acc = it & 1;
        const int nkb = k_blocks();
        if (!mbar_wait(smem_u32(&bars->acc_empty[acc]), ((acc_phase >> acc) & 1u) ^ 1u, abort_flag)) {
          if (lane == 0) report_error(err, ATENIA_ERR_DEVICE_TIMEOUT, 1200 + acc);
          *abort_flag = 1;
          ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        acc_phase ^= 1u << acc;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TN2;
        const uint32_t idesc = kInstrDesc2 | (uint32_t(tc.n >> 3) << 17);
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(smem_u32(&bars->full[stage]), phase, abort_flag)) {
            if (lane == 0) report_error(err, ATENIA_ERR_DEVICE_TIMEOUT, 1300 + stage);
            *abort_flag = 1;
            ok = false;
          }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = smem_base + stage * STAGE_BYTES2;
          tc_mma_bf16_pair_kblock(d_tmem, make_smem_desc(sa), make_smem_desc(sa + W_BYTES2), idesc, kb > 0 ? 1u : 0u);
          tc_commit_pair(smem_u32(&bars->empty[stage]));
          if (++stage == STAGES2) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) tc_commit_pair(smem_u32(&bars->acc_full[acc]));
      }
    }
  } else {
    // ================= epilogue (warps 2..9 of both CTAs) =================
    // A lane holds one weight row; the columns are token rows.  A value is stored from where it is, two bytes
    // per lane and 64 contiguous bytes per warp and token: passing the tile through shared memory for 16-byte
    // stores costs the MMAs more shared-memory cycles than it saves stores.
    // kSwiGLU: the warps of quarters q (gates) and q + 2 (ups) swap eight tokens of f32 first: the gate warp
    // finishes tokens 0..7 of a chunk of 16, the up warp tokens 8..15.
    chain_wait();
    const int quarter = warp & 3;         // TMEM lanes [32 * quarter, 32 * quarter + 32)
    const int first = ((warp - 2) >> 2);  // two warps per quarter take the 16-token chunks in turn
    float* mine = reinterpret_cast<float*>(epi + (warp - 2) * EPI_WARP_BYTES2);
    const bool up = MODE == kSwiGLU && quarter >= 2;
    // the other warp of the pair: same `first`, quarter +- 2 (warps 2..5 hold quarters 2, 3, 0, 1)
    const float* theirs = reinterpret_cast<const float*>(epi + ((warp - 2) ^ 2) * EPI_WARP_BYTES2);
    const int f_lane = (int)rank * F_CTA + (MODE == kSwiGLU ? (quarter & 1) * 32 : quarter * 32) + lane;
    const uint32_t pair_bar = 1 + first * 2 + (quarter & 1);
    int flip = 0;
    uint32_t acc_phase = 0;
    int it = 0;
    for (; seek(cur, it); ++it) {
      const int acc = it & 1;
      bool ready = mbar_wait(smem_u32(&bars->acc_full[acc]), (acc_phase >> acc) & 1u, abort_flag);
      __syncwarp();  // (each lane polled by itself; the barriers and tensor-memory loads below want the warp as one)
      if (MODE == kSwiGLU) {
        // the two warps of a pair leave together or not at all: one of them alone would hold the other in bar.sync
        uint32_t both;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 p, %1, 0;\n\t"
            "bar.red.and.pred q, %2, 64, p;\n\t"
            "selp.b32 %0, 1, 0, q;\n\t}"
            : "=r"(both)
            : "r"((uint32_t)ready), "r"(pair_bar)
            : "memory");
        ready = both != 0;
      }
      if (!ready) {
        if (lane == 0) report_error(err, ATENIA_ERR_DEVICE_TIMEOUT, 1400 + acc);
        *abort_flag = 1;
        break;
      }
      acc_phase ^= 1u << acc;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + acc * TN2;
      int ld = N;
      __nv_bfloat16* base = out;
      if constexpr (EX) {
        if (tc.group < 0) {
          ld = ex.N;
          base = ex.out;
        }
      }
      const bool f_ok = tc.f0 + f_lane < ld;
      const int t_half = up ? 8 : 0;
      __nv_bfloat16* dst = base + (size_t)(tc.row0 + t_half) * ld + tc.f0 + f_lane;
      const int rows = f_ok ? tc.rows - t_half : 0;  // tokens of the tile this lane may store
#pragma unroll 1
      for (int c = 16 * first; c < tc.n; c += 32) {
        uint32_t v[16];
        tc_ld16(taddr + c, v);
        tc_ld_wait();
        __nv_bfloat16* d = dst + (size_t)c * ld;
        if (MODE == kSwiGLU) {
          float* ex = mine + flip * 256;
#pragma unroll
          for (int j = 0; j < 8; ++j) ex[j * 32 + lane] = __uint_as_float(up ? v[j] : v[8 + j]);
          asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
          const float* ox = theirs + flip * 256;
          flip ^= 1;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float o = ox[j * 32 + lane];
            const float g = up ? o : __uint_as_float(v[j]);
            const float u = up ? __uint_as_float(v[8 + j]) : o;
            if (c + j < rows) d[(size_t)j * ld] = __float2bfloat16(silu_mul(g, u));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < rows) d[(size_t)j * ld] = __float2bfloat16(__uint_as_float(v[j]));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(mapa(smem_u32(&bars->acc_empty[acc]), 0));
    }
  }

  chain_next();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while its peer may still signal or read it
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS2)
                 : "memory");
  }
}

template <int MODE, int TOK, bool EX, typename E>
int launch_2cta_form(const GroupedGemmArgs& a, int num_sms, cudaStream_t s, const E& ex) {
  static bool attr_set[kMaxDevices] = {};
  if (first_use_on_current_device(attr_set)) {
    ATENIA_CUDA_TRY(cudaFuncSetAttribute(grouped_gemm_2cta_kernel<MODE, TOK, EX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         PairRing<TOK>::SMEM_BYTES));
  }
  const int grid = num_sms & ~1;  // whole pairs
  return launch_chained(a.chained, grouped_gemm_2cta_kernel<MODE, TOK, EX>, dim3(grid), dim3(NUM_THREADS2),
                        PairRing<TOK>::SMEM_BYTES, s, *a.pair_rows, a.tmap_b0, MODE == kSwiGLU ? a.tmap_b1 : a.tmap_b0,
                        a.group_offsets, a.num_groups, a.N, a.K, a.out, a.err, ex);
}

template <int MODE, int TOK>
int launch_2cta_one(const GroupedGemmArgs& a, int num_sms, cudaStream_t s) {
  if (a.extra.rows <= 0) return launch_2cta_form<MODE, TOK, false>(a, num_sms, s, NoExtra{});
  if constexpr (TOK == kPairTokens) {
    return ATENIA_ERR_SHAPE;  // (merges_shared: an extra group rides with tiles of at most 192 rows)
  } else {
    const PairExtra ex{*a.extra.x_rows, a.extra.tmap_b0, MODE == kSwiGLU ? a.extra.tmap_b1 : a.extra.tmap_b0, a.extra.out,
                       a.extra.rows, a.extra.N, a.extra.K};
    return launch_2cta_form<MODE, TOK, true>(a, num_sms, s, ex);
  }
}

template <int MODE>
int launch_2cta_tokens(const GroupedGemmArgs& a, int num_sms, cudaStream_t s) {
  if (a.pair_tokens == 64) return launch_2cta_one<MODE, 64>(a, num_sms, s);
  if (a.pair_tokens == 128) return launch_2cta_one<MODE, 128>(a, num_sms, s);
  if (a.pair_tokens == 192) return launch_2cta_one<MODE, 192>(a, num_sms, s);
  return launch_2cta_one<MODE, kPairTokens>(a, num_sms, s);
}

}  // namespace

int encode_pair_rows(PairRowMaps* out, const void* base, uint64_t rows, uint64_t cols, unsigned boxes) {
  int rc = ATENIA_OK;
  for (int i = 0; i < kPairBoxes && !rc; ++i)
    if (boxes >> i & 1u) rc = encode_tmap_2d_bf16(&out->box[i], base, rows, cols, pair_box_rows(i), BK);
  return rc;
}

int launch_grouped_gemm_2cta(const GroupedGemmArgs& a, int num_sms, cudaStream_t s) {
  if (a.num_groups <= 0) return ATENIA_OK;
  if (a.N % 16 != 0 || a.K % 16 != 0 || a.num_groups > kMaxGroupsShared) return ATENIA_ERR_SHAPE;
  if (!a.pair_rows) return ATENIA_ERR_NULL;
  if (a.extra.rows > 0 && (a.extra.N % 16 != 0 || a.extra.K % 16 != 0)) return ATENIA_ERR_SHAPE;
  if (a.w8) return ATENIA_ERR_UNSUPPORTED;  // INT8 weights: w8_gemm.cu / w8_gemm_m256.cu
  int rc = a.mode == kSwiGLU ? launch_2cta_tokens<kSwiGLU>(a, num_sms, s) : launch_2cta_tokens<kPlain>(a, num_sms, s);
  count_launch();
  count_tcgen05_launch();
  return rc;
}

}  // namespace atenia
