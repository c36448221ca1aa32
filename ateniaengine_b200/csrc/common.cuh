// Shared declarations of the MoE library's translation units (sm_100a only).
#pragma once
#include <vector>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/atenia_moe.h"
#include "kernel_choice.cuh"
#include "pair_tiles.cuh"

namespace atenia {

// Error word written by kernels (first error wins).  Values are the negative status codes of the
// public header; a second word keeps a site id for diagnosis.
struct DeviceError {
  int32_t code;
  int32_t site;
};

__device__ __forceinline__ void report_error(DeviceError* err, int code, int site) {
  if (err && atomicCAS(&err->code, 0, code) == 0) err->site = site;
}

// ---- bf16 helpers ---------------------------------------------------------------------------
__device__ __forceinline__ float bf16_bits_to_f32(uint32_t b) { return __uint_as_float(b << 16); }
__device__ __forceinline__ float bf16lo(uint32_t packed) { return __uint_as_float(packed << 16); }
__device__ __forceinline__ float bf16hi(uint32_t packed) { return __uint_as_float(packed & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// ---- launch bookkeeping ---------------------------------------------------------------------
void count_launch(int n = 1);
void count_tcgen05_launch();
void count_bytes(int which, uint64_t n);

// One-time kernel attributes are per device: `flags` is a per-kernel array indexed by device ordinal.
// Returns true exactly once per (kernel, device); a benign double set under a race is harmless.
constexpr int kMaxDevices = 64;
inline bool first_use_on_current_device(bool (&flags)[kMaxDevices]) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return true;
  if (flags[dev]) return false;
  flags[dev] = true;
  return true;
}

// ---- chained launches --------------------------------------------------------------------------
// The kernels of a forward are launched so that each may start while the one before it on the stream still runs
// (programmatic dependent launch).  Every kernel launched with launch_chained therefore calls chain_wait() before it
// touches global memory at all: it returns once the kernel before has completed and its stores are visible -- and that
// one's chain_wait() has waited for the kernel before it, so nothing earlier is in flight either.  chain_next() lets
// the next kernel's blocks start: what overlaps is its launch, not its work.  Kernels without chain_wait() are
// launched plainly and wait for everything before them as usual.
// Two exceptions.  The cluster router requests rows of the layer's own copies of the router matrix and the gate vector, which
// no kernel writes (set_weights synchronises).  And a GEMM takes the group offsets and requests its first weight tiles before
// its chain_wait().  The kernel before it writes neither (it gathers rows, makes digits, or is the GEMM before) and comes to
// chain_next() only past its own chain_wait() -- or, between two GEMMs, was launched by one that had passed its -- so
// whatever wrote them has completed before the GEMM's blocks start.  Under expert parallelism every kernel of ep.cu is launched
// plainly and calls no chain_next(), and one of them (the scatter, or the host's read of the counts) comes between the kernel
// that writes the offsets and the GEMM, whatever the collective right before it does.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// A kernel that takes whole SMs must not sit there waiting while another stream's work could run.  So the kernels
// before the first GEMM of a forward (row gather, digit quantiser) call chain_next() after their chain_wait(): the GEMM
// comes no earlier than the rows it reads are being written, and not already beside the router (one token of the
// Mixtral shape 137.3 -> 134.8 us for it, other sizes the same).  Beside a layer's own shared expert the GEMMs are
// not chained at all (`chained` false: Qwen1.5-MoE shape, 2048 tokens, in bursts after a pause, 342 -> 372 us when the
// routed GEMM displaced the shared expert's).  A captured launch becomes a programmatic edge of the graph (eight INT8
// layers, 8 tokens: 1609 -> 1573 us one graph after another, 1413 -> 1365 with three on their streams).  Two layers on
// two streams, in all ms for the same calls, chained / plain: Mixtral shape of 1024 tokens beside a 64-expert layer of 64
// 44.2 / 46.7, 4096 beside 64 42.5 / 49.2, 64 beside 16 33.5 / 35.6.
// ATENIA_MOE_CHAINED=0 makes every launch of a layer plain.
template <typename... P, typename... A>
int launch_chained(bool chained, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) (void)cudaGetLastError();  // returned here: not again by the next plain launch's check
  return (int)e;
}

#define ATENIA_CUDA_TRY(expr)                \
  do {                                       \
    cudaError_t e__ = (expr);                \
    if (e__ != cudaSuccess) return (int)e__; \
  } while (0)

// ---- router / routing ------------------------------------------------------------------------
struct RouterArgs {
  const void* x;          // [T, d] bf16 or f32
  int x_is_f32;
  const float* w_router;  // [E, d] f32
  const float* bias;      // [E] or null
  const float* gate_vec;  // [d] or null
  int T, d, E, k, renormalize;
  int32_t* topk_idx;   // [T, k]
  float* topk_w;       // [T, k]
  float* gate_scale;   // [T] or null
  float* logits;       // [T, E] or null
  DeviceError* err;
  int variant;         // -1: by size; 0: CUDA-core f64 kernel (router.cu); 1: f64 tensor-core kernel
                       // (router_dmma.cu); 2: split-k kernel (router_splitk.cu) up to kSplitkPinnedTokens;
                       // 3: integer router (router_i8.cu) wherever it can serve the call, else by size
  const CUtensorMap* digit_map;  // integer router (router_i8.cu): digit planes of the router matrix (host pointer; null: the
  const double* digit_scale;     // layer has none that hold it exactly) and the scale of each of its rows (NaN: row not held)
  bool chained;        // see launch_chained
  bool beside;         // a shared expert's GEMMs run on another stream meanwhile
};
int launch_router(const RouterArgs& a, cudaStream_t s);
int launch_router_dmma(const RouterArgs& a, cudaStream_t s);  // same contract, E <= 128, k <= 8
int launch_router_splitk(const RouterArgs& a, cudaStream_t s);  // same contract
bool router_splitk_pays(int T, int E, int d, bool beside);
constexpr int kSplitkPinnedTokens = 1024;
// Integer router of bf16 activations: layers of at most 64 rows of w (experts, and the gate vector if the call wants it).
// planes [kRouterDigitPlanes][kRouterDigitRows][d] int8, map with box {128, kRouterDigitPlanes * kRouterDigitRows / 2} and
// the 128-byte swizzle; scale [kRouterDigitRows].
constexpr int kRouterDigitRows = 64, kRouterDigitPlanes = 5;
constexpr int kRouterDigitMaxK = 16384;  // (int32 sums of up to four products of 2^14 a k)
// Does a layer get the planes?  (16 experts or fewer: the f64 routers are as fast)
inline bool router_digits_built(int E, int d) { return E > 16 && E <= kRouterDigitRows && d <= kRouterDigitMaxK; }
int launch_router_i8(const RouterArgs& a, cudaStream_t s);
int launch_router_digits(const float* router, const float* gate, int E, int d, int8_t* planes, double* scale, cudaStream_t s);
int launch_route_from_logits(const float* logits, int T, int E, int k, int renormalize,
                             int32_t* topk_idx, float* topk_w, DeviceError* err, cudaStream_t s);

// DeepSeek-V3 routing from logits (one thread per token runs v3_route_one of v3_route.cuh).
int launch_v3_route(const float* logits, const float* e_score_bias, int T, int E, int k, int n_group, int topk_group,
                    int norm_topk_prob, float scaling, int32_t* topk_idx, float* topk_w, DeviceError* err,
                    cudaStream_t s);

// ---- dispatch --------------------------------------------------------------------------------
struct DispatchArgs {
  const int32_t* topk_idx;  // [n] flat (t*k + s) -> expert
  int n;                    // T * k
  int E;
  int32_t* block_counts;  // [E, nblk] entries of each expert per block of kDispatchChunk entries
  int32_t* block_base;    // [E, nblk] exclusive scan of block_counts over the blocks
  int32_t* expert_offsets;  // [E + 1]
  int32_t* perm;            // [n]
  int32_t* inv_perm;        // [n]
  int32_t* extra_offsets;   // [2] = {0, T} for the shared-expert group, or null
  int T;
  DeviceError* err;
  bool chained;  // see launch_chained
};
constexpr int kDispatchChunk = 256;  // flat entries per block
int launch_dispatch(const DispatchArgs& a, cudaStream_t s);

// x_perm[r, :] = bf16(x[perm[r] / k, :]) for r < *placed (device: expert_offsets[E], the rows the
// placement wrote); optionally x_bf16 = bf16(x) when x is f32.
int launch_gather_rows(const void* x, int x_is_f32, const int32_t* perm, const int32_t* placed, int n_rows, int k,
                       int d, __nv_bfloat16* x_perm, __nv_bfloat16* x_bf16, int T, bool chained, cudaStream_t s);

// ---- combine ---------------------------------------------------------------------------------
struct CombineArgs {
  const __nv_bfloat16* y_rows;  // [n, d] expert outputs in dispatch order
  const int32_t* inv_perm;      // [T*k]
  const float* topk_w;          // [T*k]
  const __nv_bfloat16* y_shared;  // [T, d] or null
  const float* gate_scale;        // [T] or null (null = 1.0)
  const float* residual;          // [T, d] f32 added last, or null (layer stacks)
  void* out;
  int out_is_f32;
  int T, k, d;
  bool chained;  // see launch_chained: nothing but kernels of this stream before it
};
int launch_combine(const CombineArgs& a, cudaStream_t s);

// ---- grouped GEMM ----------------------------------------------------------------------------
// One "group" is a contiguous block of rows of A multiplied by that group's own weight matrices.
//   kSwiGLU: out[r, n] = silu(A[r,:].B0_g[n,:]) * (A[r,:].B1_g[n,:])      (gate / up, N = d_ff)
//   kPlain:  out[r, n] = A[r,:].B0_g[n,:]                                   (down, N = d_model)
// B matrices are row-major [N, K] (K contiguous): the reference's weight layout.
enum GemmMode { kSwiGLU = 0, kPlain = 1 };

// Token rows of the CTA-pair kernel: the same buffer in boxes of several heights (pair_tiles.cuh).
struct PairRowMaps {
  CUtensorMap box[kPairBoxes];
};

struct GroupedGemmArgs {
  CUtensorMap tmap_a;              // A [rows_cap, K] bf16, box {64, 128}, 128B swizzle
  const CUtensorMap* tmap_b0;      // device array [num_groups]
  const CUtensorMap* tmap_b1;      // device array [num_groups] (kSwiGLU only)
  const int32_t* group_offsets;    // device [num_groups + 1] row offsets into A / out
  int num_groups;
  int N, K;
  int mode;
  __nv_bfloat16* out;  // [rows_cap, N]
  // INT8 weights: per-group device pointers to f32 per-row scales (null for bf16)
  const float* const* scale0;  // device array [num_groups] of device pointers
  const float* const* scale1;
  DeviceError* err;
  int max_rows;  // upper bound on total rows (sizes nothing; used by the checking kernel's grid)
  const PairRowMaps* pair_rows;  // CTA-pair kernel only (host pointer, copied at the launch)
  int pair_tokens;  // ... token rows of a tile at most: 64, 128, 192, else 256 (pair_tokens_of)
  // CTA-pair kernel only: one more group in the same launch, with its own matrices, rows, sizes and output (the shared
  // expert beside the routed ones).  rows 0: none.
  struct Extra {
    const PairRowMaps* x_rows;  // host pointer, copied at the launch
    const CUtensorMap* tmap_b0;
    const CUtensorMap* tmap_b1;
    __nv_bfloat16* out;
    int rows, N, K;
  } extra;
  int w8;        // B matrices are int8 (tensor maps of bytes), widened to bf16 inside the kernel
  float* splitk_ws;  // W8 tensor-memory kernel: workspace for stream-K partial sums (null: whole tiles only)
  // stream-K decode kernels: zeroed counters [kSplitKMaxTiles * 8] with which the kernel finishes the split
  // tiles itself (null: a second kernel adds the pieces)
  unsigned int* splitk_cnt;
  // integer-MMA decode kernel only: 2^(e - 26) per token row and the row count of one digit plane
  const float* tok_scale;
  int plane_rows;
  bool chained;  // see launch_chained
};
int launch_grouped_gemm_tcgen05(const GroupedGemmArgs& a, int num_sms, cudaStream_t s);

// Plain CUDA-core version of the same contraction, reading the same buffers through ordinary
// pointers.  Used by the test-suite to localise a fault; never selected by the forward path.
struct GroupedGemmCheckArgs {
  const __nv_bfloat16* a;  // [rows, K]
  const void* const* b0;   // device array [num_groups] of device pointers to [N, K]
  const void* const* b1;
  int b_is_int8;
  const float* const* scale0;
  const float* const* scale1;
  const int32_t* group_offsets;
  int num_groups, N, K, mode;
  __nv_bfloat16* out;
  int max_rows;
  bool chained;  // matrix-vector kernel: see launch_chained
};
int launch_grouped_gemm_check(const GroupedGemmCheckArgs& a, cudaStream_t s);
// The same contraction for calls of at most two rows in all (decode at batch 1): a CUDA-core
// matrix-vector kernel that streams the touched experts' weights once (decode_gemv.cu; it handles up to
// four rows per group, but from three rows on the tensor-core kernels are as fast).
int launch_grouped_gemv(const GroupedGemmCheckArgs& a, cudaStream_t s);
constexpr int kGemvMaxRows = 2;
// rows x d x F above which a bf16 call of at most kGemvMaxRows rows takes the stream-K kernel instead.  One token,
// top-2 of 8 experts on a B200, matrix-vector / stream-K: d 4096, F 3584 66.0 / 69.3 us, F 7168 97.3 / 97.8,
// F 14336 157.3 / 147.4.
constexpr int64_t kGemvMaxWeights = (int64_t)1 << 26;

int launch_f32_to_bf16(const float* src, __nv_bfloat16* dst, int64_t n, cudaStream_t s);
// p[0] = a, p[1] = b on the stream (the one-group offsets of the shared expert's GEMMs)
int launch_set_pair(int32_t* p, int32_t a, int32_t b, cudaStream_t s);
// y = (x * inv_rms(x)) * gamma per row (stack.cu); gamma may be null (unit gain)
int launch_rmsnorm_rows(const float* x, const float* gamma, float eps, float* y, int T, int d, bool chained,
                        cudaStream_t s);

// Tensor-map encoding through the driver entry point (no link-time dependency on libcuda).
int encode_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols,
                        uint32_t box_rows, uint32_t box_cols);
// grouped_gemm_2cta.cu; `boxes` (bit i: box i) are encoded, a launch reads no others
int encode_pair_rows(PairRowMaps* out, const void* base, uint64_t rows, uint64_t cols, unsigned boxes = kPairAllBoxes);
// int8 matrix [rows, cols]; unswizzled box, or 64-byte swizzle for the row-per-thread reads of the
// TMEM-operand kernel
int encode_tmap_2d_u8(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows,
                      uint32_t box_cols, int swizzle64);  // swizzle64: 0 none, 1 64-byte, 2 128-byte
// W8A16 grouped GEMM with the weights as the tensor-memory operand (w8_gemm.cu).  tmap_a is the bf16
// token matrix (box {64, 128}, 128B swizzle); tmap_b0/b1 are int8 maps with the 64-byte swizzle.
int launch_grouped_gemm_w8_tmem(const GroupedGemmArgs& a, int num_sms, cudaStream_t s);
constexpr size_t kW8SplitKSlotFloats = 2 * 128 * 128;  // per CTA: two slots of this size
constexpr int kSplitKMaxTiles = 8 * 160;               // tiles a stream-K launch can have (eight rounds of the SMs)
// W8A16 for large groups (w8_gemm_m256.cu): 256-row token tiles, the widened weight tile shared by two
// M128 MMAs.  Tensor maps as for launch_grouped_gemm_tcgen05 with w8 set.
int launch_grouped_gemm_w8_m256(const GroupedGemmArgs& a, int num_sms, cudaStream_t s);
// bf16 weights, groups of at most 128 rows (bf16_decode_gemm.cu): transposed product with stream-K over
// the SMs; tmap_a / tmap_b0 / tmap_b1 are the maps of launch_grouped_gemm_tcgen05, splitk_ws as for
// the INT8 tensor-memory kernel (null: whole tiles only).
int launch_grouped_gemm_bf16_decode(const GroupedGemmArgs& a, int num_sms, cudaStream_t s);
// INT8 weights, calls of at most kI8DecodeMaxRows rows (same file): the codes are multiplied as integers
// (tcgen05 kind::i8) with the token rows split into four planes of base-128 digits by
// launch_quantize_digits.  tmap_a is the digit-plane map (uint8, box {128, 16}, 128B swizzle; plane p of
// row r at row p * plane_rows + r), tmap_b0 / tmap_b1 int8 maps with box {128, 128} and the 128B swizzle.
constexpr int kI8DecodeMaxRows = 512;      // largest call (rows of one digit plane) a layer may be set up for
// ... and what it is set up for unless told otherwise (512 rows of the Mixtral shape: 526 us, tensor-memory kernel 391).
// Which calls take it up to there: i8_decode_pays (kernel_choice.cuh).
constexpr int kI8DecodeDefaultRows = 256;
int launch_grouped_gemm_w8_i8_decode(const GroupedGemmArgs& a, int num_sms, cudaStream_t s);
// planes [4][plane_rows][K] int8 and tok_scale [plane_rows] of n_rows rows; n_rows_dev (device, may be null)
// bounds the rows that hold data.  Row r comes from row r of src.x, or -- with src.perm, the dispatch
// permutation -- from token row perm[r] / k of the caller's batch (the row gather and the digits in one pass).
// `between`: the launch before is the layer's first GEMM (the second may then be launched early).
struct DigitSource {
  const void* x;        // [n_src_rows, K], bf16 or f32
  int x_is_f32;
  const int32_t* perm;  // null: no gather
  int k;
  int n_src_rows;
};
int launch_quantize_digits(const DigitSource& src, const int32_t* n_rows_dev, int n_rows, int K, int plane_rows,
                           int8_t* planes, float* tok_scale, bool between, bool chained, cudaStream_t s);
// bf16 weights, CTA pairs (tcgen05 cta_group::2), transposed product: pair_rows describes the token rows (tmap_a
// is not read), tmap_b0 / tmap_b1 have boxes of kPairWeightRows (kSwiGLU) or 128 (kPlain) weight rows
constexpr int kPairWeightRows = 64;
inline int pair_f_tiles(int n, int mode) { return mode == kSwiGLU ? (n + 127) / 128 : (n + 255) / 256; }  // feature tiles
int launch_grouped_gemm_2cta(const GroupedGemmArgs& a, int num_sms, cudaStream_t s);
// bf16 weights, CTA pairs, token rows as the M side (grouped_gemm_pair_rows.cu): tensor maps of the single-CTA kernel
int launch_grouped_gemm_pair_rows(const GroupedGemmArgs& a, int num_sms, cudaStream_t s);

// Sub-batch sizes for the host-buffer operator (planner.cu): n tokens in pieces of at most cap tokens,
// chosen with a cost model of the copies and the forward; one piece means "do not overlap".  `fit`
// (optional) carries what the operator measured in its earlier calls: forward(T) = a + b T milliseconds
// and the copy time of a token.
struct ExecFit {
  double a_ms = 0.0, b_ms = 0.0, copy_token_ms = 0.0;
  bool valid = false;
};
std::vector<uint64_t> plan_exec_pieces(const AteniaMoeConfig& c, uint64_t n, uint64_t cap, const ExecFit* fit);
double model_exec_ms(const AteniaMoeConfig& c, const std::vector<uint64_t>& pieces, const ExecFit* fit);
void update_exec_fit(const AteniaMoeConfig& c, const uint64_t* tokens, const float* forward_ms, int n_pieces,
                     uint64_t copy_tokens, float copy_ms, ExecFit* fit);

}  // namespace atenia
