// Host-callable launchers of the CUDA kernels (implemented in the .cu files). All launch on the
// given stream and return the cudaError_t of the launch. Pointers are device pointers.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "common.h"

namespace etc {

// ---- f16 activation hand-off ------------------------------------------------------------------
// Activations travel between the kernels of an invocation as f16 in the tensor cores' operand order: [chunk of nv rows]
// [K/8][nv][8] with nv = hand_off_stride(rows) = 32, 64 or 128; only 128 has more than one chunk.
inline int hand_off_stride(int64_t rows) { return rows <= 32 ? 32 : (rows <= 64 ? 64 : 128); }
// Rows padded to whole chunks: the size of a buffer that any number of rows up to `rows` fits.
inline int64_t hand_off_rows(int64_t rows) { return rows <= 64 ? hand_off_stride(rows) : (rows + 127) / 128 * 128; }
// Offset (in halves) of columns 8 * k8 .. 8 * k8 + 7 of a row of k8_total * 8 columns.
__host__ __device__ inline size_t hand_off_cell(int k8, size_t row, int nv, int k8_total) {
  const int shift = nv == 32 ? 5 : (nv == 64 ? 6 : 7);
  return ((((row >> shift) * k8_total + k8) << shift) + (row & (nv - 1))) * 8;
}

// ---- block-quantized weights (quant_kernels.cu) ------------------------------------------
cudaError_t launch_dequantize(int codec, const uint8_t* packed, int64_t rows, int64_t columns, float* out,
                              cudaStream_t stream);
cudaError_t launch_quantize(int codec, const float* x, int64_t rows, int64_t columns, uint8_t* packed,
                            cudaStream_t stream);
cudaError_t launch_qlinear_generic(int codec, const float* x, int64_t vectors, int64_t columns, const uint8_t* weight,
                                   int64_t rows, const float* bias, float* out, int sm_count, cudaStream_t stream, int* launches, int64_t out_stride = 0);
cudaError_t launch_qembedding(int codec, const void* indexes, int index_is_i64, int64_t count, const uint8_t* weight,
                              int64_t rows, int64_t columns, float* out, DeviceStatus* status, cudaStream_t stream);

// Tiled weights: 128-row tiles, rows padded with zero scales. For row tile t and 32-column block kb the 128 rows' payloads are
// contiguous ([tile][block][row][bytes]), 16 bytes of 4-bit codes (Q4_0, Q4_K; nibbles placed so that masks give f16
// pairs in column order, see dequant.cuh) or 32 bytes of 8-bit ones (Q8_0 and the re-cut Q3_K, Q5_K, Q6_K). Scales are [tile][block][row], one
// f16 (Q4_0, Q8_0: the byte count of the GGUF encoding) or two (K-quants: scale and minimum, or the scales of the two
// halves). Both linear kernels (qlinear_stream.cu, qlinear_umma.cu) read this one layout.
//
// A run of 128-row tiles of one codec inside a tiled weight. A weight fused from parts of different codecs (q and k in
// Q4_K, v in Q6_K, as GGUF files mix them) holds one segment per run of equal codecs, each repacked in its codec's layout
// at byte offsets into the weight's arrays; the linear launches one kernel per segment into the same outputs.
struct TiledSegment {
  int codec = 0;
  int tile0 = 0, tiles = 0;
  size_t quant_offset = 0, scale_offset = 0;  // bytes
};
constexpr int kMaxSegments = 4;

struct TiledWeight {
  int codec = 0;            // the first segment's codec
  int64_t rows = 0;         // logical rows (outputs) after concatenation / interleave
  int64_t rows_padded = 0;  // multiple of 128
  int64_t columns = 0;      // multiple of 64
  int interleave8 = 0;
  uint8_t* quants = nullptr;
  __half* scales = nullptr;
  size_t quant_bytes = 0, scale_bytes = 0;
  int n_segments = 0;       // 0: one segment of `codec` over the whole weight
  TiledSegment segments[kMaxSegments];
};
// Split-K partials a linear left unsummed for the kernel that consumes its result (the next RMSNorm, or the RoPE /
// KV-append kernel): [splits][vpad][rows_padded] f32, summed in split order. splits == 0: the result is already in `out`.
struct DeferredSum {
  const float* partials = nullptr;
  int splits = 0, vpad = 0, rows_padded = 0;
};

struct RepackParts {
  const uint8_t* ptr[4];
  int64_t rows[4];
  int n_parts;
};
cudaError_t launch_repack(const TiledWeight& w, const RepackParts& parts, cudaStream_t stream);

// f32 [vectors, K] to the hand-off layout with row stride nv (16, 32, 64 or 128), absent vectors zero.
cudaError_t launch_hand_off_convert(const float* x, int64_t vectors, int K, int nv, __half* xh, int sm_count, cudaStream_t stream);

// Sums split-K partials [chunk of vpad vectors][splits][vpad][rows_padded] in split order and runs the epilogue.
cudaError_t launch_qlinear_reduce(const float* scratch, int splits, int vpad, int vectors, int rows, int rows_padded,
                                  const float* bias, const float* residual, int epilogue, float* out, __half* out_xh, int xh_nv, cudaStream_t stream);

// decode batches up to stream_max_vectors() (qlinear_stream.cu)
struct StreamPlan {
  int nv = 32;                  // vectors padded to the MMA N (16, 32, 64 or 128)
  int tiles = 1, stages = 1;    // 128-row tiles, stages of four 32-value blocks per tile
  int splits = 1, stages_per_split = 1;  // CTAs that share a tile's K: a cluster, or with `deferred` writers of partial sums
  bool deferred = false;
  size_t xh_bytes = 0;          // f16 activations, at the head of the scratch (rounded to 256 bytes)
  size_t scratch_bytes = 0;     // partial sums behind them
};
StreamPlan plan_stream(const TiledWeight& w, int64_t vectors, int sm_count, bool deferred);
int stream_max_vectors();
size_t stream_scratch_bytes(const TiledWeight& w, int64_t vectors, int sm_count);
// x f32 [vectors, K], or xh_ready in the f16 hand-off layout with row stride xh_nv.
cudaError_t launch_qlinear_stream(const TiledWeight& w, const float* x, const __half* xh_ready, int64_t vectors, const float* bias,
                                  const float* residual, int epilogue, float* out, __half* out_xh, void* scratch, DeviceStatus* status,
                                  int sm_count, cudaStream_t stream, int* launches, int xh_nv = 32, DeferredSum* defer = nullptr);

// prefill and large batches (qlinear_umma.cu)
struct UmmaPlan {
  int nv = 128;              // vectors per chunk (the MMA N)
  int chunks = 1, tiles = 1, stages = 1;  // 128-row tiles, stages of four 32-value blocks per tile
  int splits = 1, stages_per_split = 1;
  size_t xh_bytes = 0;       // f16 activations in [chunk][K/8][nv][8] order, all chunks
  size_t scratch_bytes = 0;  // split-K partials [chunk][split][nv][rows_padded], all chunks
};
UmmaPlan plan_umma(const TiledWeight& w, int64_t vectors, int sm_count);
// x: f32 [vectors, K], converted to f16 in xh first, or xh_ready in the hand-off layout.
cudaError_t launch_qlinear_umma(const TiledWeight& w, const float* x, const __half* xh_ready, int64_t vectors, const float* bias,
                                const float* residual, int epilogue, float* out, __half* out_xh, __half* xh, float* scratch, DeviceStatus* status, int sm_count, cudaStream_t stream,
                                int* launches);

// Front end of the tiled linear. `scratch` must hold tiled_scratch_bytes(w, vectors, sm_count).
size_t tiled_scratch_bytes(const TiledWeight& w, int64_t vectors, int sm_count);
// xh_ready / out_xh: optional f16 activation hand-off between kernels with xh_nv = hand_off_stride(vectors).
cudaError_t launch_qlinear_tiled(const TiledWeight& w, const float* x, int64_t vectors, const float* bias,
                                 const float* residual, int epilogue, float* out, void* scratch, DeviceStatus* status,
                                 int sm_count, cudaStream_t stream, int* launches, const __half* xh_ready = nullptr,
                                 __half* out_xh = nullptr, int xh_nv = 32, DeferredSum* defer = nullptr);
// RMSNorm whose output is stored in the hand-off layout, after x += the sum of a projection's split-K partials where
// sum.splits > 0 (x, the residual stream, is updated in place).
cudaError_t launch_sum_rmsnorm_xh8(float* x, const DeferredSum& sum, const float* weight, double eps, int64_t rows, int64_t n,
                                   __half* out_xh, cudaStream_t stream, int xh_nv);

// ---- tensor-parallel all-reduce over peer memory (tp_kernels.cu) -----------------------------
constexpr int kMaxTpRanks = 8;
// One rank's exchange region: [0, 96) three flag arrays of kTpFlagStride words (partial sums stored, slice totals stored,
// picks stored), [256, 288) counters private to the owner, [1024, 1024 + 8 * kTpMaxPicks) (best logit, token) pairs, then
// from kTpHeaderBytes on two exchange buffers of (world + 1) slots of `slot_bytes` each: an inbox with one slot per
// sender, and the table of totals.
constexpr int kTpFlagStride = 8;
constexpr size_t kTpCounterOffset = 256, kTpPickOffset = 1024, kTpHeaderBytes = 4096;
constexpr int kTpMaxPicks = 256;
constexpr long long kTpWaitCycles = 1ll << 31;  // about a second
struct PeerView {
  float* inbox[kMaxTpRanks][2];   // every rank's inboxes [world][slot] (own: local memory, others: peer mappings)
  float* totals[kMaxTpRanks][2];  // every rank's tables of slice totals [slot]
  uint32_t* flags[kMaxTpRanks];   // every rank's flag arrays; entry r of each is written by rank r
  uint2* picks[kMaxTpRanks];      // every rank's (best logit bits, token) per lane
  int rank, world;
};
inline size_t tp_slot_bytes(size_t capacity_floats) { return (capacity_floats * sizeof(float) + 255) & ~(size_t)255; }
inline size_t tp_region_bytes(size_t capacity_floats, int world) {
  return kTpHeaderBytes + 2 * (size_t)(world + 1) * tp_slot_bytes(capacity_floats);
}
inline void tp_view_bind(PeerView& view, int r, unsigned char* base, size_t slot_bytes, int world) {
  view.flags[r] = reinterpret_cast<uint32_t*>(base);
  view.picks[r] = reinterpret_cast<uint2*>(base + kTpPickOffset);
  for (int b = 0; b < 2; ++b) {
    unsigned char* buffer = base + kTpHeaderBytes + (size_t)b * (world + 1) * slot_bytes;
    view.inbox[r][b] = reinterpret_cast<float*>(buffer);
    view.totals[r][b] = reinterpret_cast<float*>(buffer + (size_t)world * slot_bytes);
  }
}
// hidden[0, count) += sum over ranks of their partial sums; count is a multiple of 4. This rank's partial sum is
// `partial`, or with sum.splits > 0 the sum of the split-K partials of a [count / columns, columns] projection result.
cudaError_t launch_tp_allreduce(const PeerView& view, int buffer, float* hidden, size_t count, int columns, const DeferredSum& sum,
                                const float* partial, bool two_shot, uint32_t* counters, long long wait_cycles, int sm_count,
                                DeviceStatus* status, cudaStream_t stream);
// tokens[b] = the token of the largest logit over all ranks' picks (lowest token on ties), b < batch <= kTpMaxPicks.
cudaError_t launch_tp_pick(const PeerView& view, int batch, uint32_t* tokens, uint32_t* counters, long long wait_cycles,
                           DeviceStatus* status, cudaStream_t stream);

// ---- dense / elementwise (elementwise.cu) --------------------------------------------------
// Dense f32 linear(s) over one input: out[p][row, col] = x W[p]^T for up to three weights of one launch, all with row stride
// out_stride. `residual` (same layout as the one output) is added; `swiglu`: two weights of n[0] rows, silu(gate) * up.
struct DenseArgs {
  const float* x = nullptr;
  int64_t m = 0, k = 0;
  const float* w[3] = {};
  int64_t n[3] = {};
  float* out[3] = {};
  int64_t out_stride = 0;
  int parts = 1;
  const float* bias = nullptr;      // parts == 1 only
  const float* residual = nullptr;  // parts == 1 only
  int swiglu = 0, exact = 0;
  int constant_weights = 0;         // no earlier kernel of the stream writes the weights: they are fetched ahead of it
  const float* norm_weight = nullptr;  // x goes through RMSNorm on the way; only where dense_norm_rides
  double norm_eps = 0.0;
  int sm_count = 1;
};
bool dense_narrow_supported(const DenseArgs& a);  // few rows, 32 weight rows and all inputs in shared memory, and faster than the ring
bool dense_norm_rides(const DenseArgs& a, int64_t tiles);  // of a launch with that many tiles of 32 weight rows
bool dense_linear_supported(const DenseArgs& a);  // k a multiple of 4, 16-byte aligned operands
cudaError_t launch_dense_linear(const DenseArgs& a, cudaStream_t stream);
cudaError_t launch_linear_f32(const float* x, int64_t m, int64_t k, const float* w, int64_t n, const float* bias,
                              float* out, int sm_count, cudaStream_t stream);
cudaError_t launch_rmsnorm(const float* x, const float* weight, double eps, int64_t rows, int64_t n, float* out,
                           cudaStream_t stream);
cudaError_t launch_rope(const float* x, const int64_t* offsets, int64_t n_offsets, const double* inv_freq, int layout,
                        int64_t batch, int64_t heads, int64_t steps, int64_t head_dim, float* out, cudaStream_t stream);
cudaError_t launch_swiglu(const float* gate, const float* up, int64_t n, float* out, int exact, cudaStream_t stream);
cudaError_t launch_add(const float* a, const float* b, int64_t n, float* out, cudaStream_t stream);
cudaError_t launch_argmax(const float* logits, int64_t rows, int64_t vocab, uint32_t* tokens, DeviceStatus* status,
                          cudaStream_t stream,
                          uint2* picks = nullptr, uint32_t index_base = 0, uint32_t* mirror = nullptr);
// One token per logits row by temperature / top-k / top-p sampling with the splitmix64 draw (sampling.cu); temperature
// must be positive here (zero is the argmax kernel's case). seeds / counters: optional per-row device arrays.
cudaError_t launch_sample_rows(const float* logits, int64_t rows, int64_t vocab, double temperature, int64_t top_k, double top_p,
                               uint64_t seed, uint64_t counter, const uint64_t* seeds, const uint64_t* counters, uint32_t* tokens,
                               DeviceStatus* status, cudaStream_t stream);
cudaError_t launch_embedding_f32(const void* indexes, int index_is_i64, int64_t count, const float* table, int64_t rows,
                                 int64_t columns, float* out, DeviceStatus* status, cudaStream_t stream);
// Copy row (advance-1) of each lane's [T, width] block into [lanes, width] (LastTokenRow).
cudaError_t launch_last_token_rows(const float* src, int64_t lanes, int64_t steps, int64_t width, int64_t advance,
                                   float* out, cudaStream_t stream);

// ---- paged KV (attention.cu) -----------------------------------------------------------------
// Device pool geometry. Page-major layout chosen for the B200: each (page, kv head) holds its
// block_size token rows contiguously: elem(page, head, slot, d) = ((page*kv_heads + head)*block_size + slot)*head_dim + d.
struct PoolView {
  void* k = nullptr;       // this layer's K slab
  void* v = nullptr;
  float* k_scale = nullptr;  // u8 tier: [page][head][slot]
  float* v_scale = nullptr;
  int dtype = 0, kv_heads = 0, head_dim = 0, block_size = 0;
};
// Per-lane step description in device memory.
struct LaneInfo {
  int cursor;      // tokens already committed
  int advance;     // live query rows in this step (0 = padded lane)
  int start;       // first position still resident (pool window), 0 without
  int table_offset;  // offset of this lane's block table in the tables array (index 0 = block of position 0)
};
cudaError_t launch_kv_append(const PoolView& pool, const float* k, const float* v, const LaneInfo* lanes,
                             const int* tables, int batch, int tokens, int64_t lane_stride, int64_t head_stride,
                             int64_t token_stride, cudaStream_t stream);
// Reference-order attention in f64 (any tier, any block size, window). q/out [B,Hq,T,D] f32, or [B,T,Hq,D].
// scratch: f64 [B*Hq*T][max_ctx]. op_window < 0: none.
cudaError_t launch_attention_exact(const PoolView& pool, const float* q, const LaneInfo* lanes, const int* tables,
                                   int batch, int q_heads, int tokens, double scale, long long op_window, float* out,
                                   double* scratch, int max_ctx, cudaStream_t stream, bool tokens_first = false);
// Tensor-core flash-decoding over the block table (f16/bf16 tiers, block_size 16, head_dim 64/128,
// one query token per lane). q [B,Hq,D] f32; out [B,Hq,D] f32. partial scratch for splits > 1.
struct AttnPlan {
  int splits = 1;
  int pages_per_split = 0;
  size_t scratch_bytes = 0;
  int sm_count = 1;
};
AttnPlan plan_attention(int batch, int q_heads, int kv_heads, int head_dim, int max_pages, int sm_count);
// Largest scratch plan_attention can ask for with tables of at most max_pages pages.
size_t plan_attention_max_scratch(int batch, int q_heads, int kv_heads, int head_dim, int max_pages, int sm_count);
bool attention_mma_supported(const PoolView& pool, int q_heads, int tokens);
// For a decode step: q is not given but comes from the fused projection's rows (or their partials), RoPE and the append of the
// new token's K and V happen in the attention kernel. Everything else that the kernel reads (cached rows, lanes, tables) must
// have been written before the launches of this step.
struct FusedRope {
  const float* qkv;
  DeferredSum sum;
  const double* inv_freq;
  int layout;
};
cudaError_t launch_attention_mma(const PoolView& pool, const float* q, const LaneInfo* lanes, const int* tables,
                                 int batch, int q_heads, double scale, long long op_window, float* out,
                                 const AttnPlan& plan, float* scratch, cudaStream_t stream, int* launches,
                                 __half* out_xh = nullptr, int xh_nv = 32, int tokens = 1, const FusedRope* rope = nullptr);
// RoPE, append and reference-order attention of a decode step (f32 cache, contexts of at most max_ctx in shared memory). As with
// FusedRope, all it reads but qkv must have been written before the launches of this step.
bool attention_exact_step_supported(const PoolView& pool, int batch, int q_heads, int max_ctx, int sm_count);
cudaError_t launch_attention_exact_step(const PoolView& pool, const float* qkv, const LaneInfo* lanes, const int* tables, const double* inv_freq, int layout,
                                        int batch, int q_heads, double scale, long long op_window, float* out, int max_ctx, cudaStream_t stream);
// Fused RoPE(q), RoPE(k) and KV append: qkv [B * tokens, (Hq+2*Hkv)*D] f32 (the fused projection output) ->
// q_out [B, tokens, Hq, D] f32 rotated, K/V rows written to the pool at positions cursor .. cursor + tokens - 1.
cudaError_t launch_rope_append(const PoolView& pool, const float* qkv, const LaneInfo* lanes, const int* tables,
                               const double* inv_freq, int layout, int batch, int q_heads, float* q_out,
                               cudaStream_t stream, const DeferredSum* sum = nullptr, int tokens = 1);
// Tail of a device-resident greedy step: feeds the sampled tokens back as the next ids, appends
// them to the history, and advances every live lane's cursor (and window start) by one.
cudaError_t launch_record_step(const uint32_t* tokens, uint32_t* ids, uint32_t* history, int* step_counter, LaneInfo* lanes,
                               int batch, long long window, cudaStream_t stream);
cudaError_t launch_pool_read_rows(const PoolView& pool, const uint32_t* rows, int64_t n, float* out, int which,
                                  cudaStream_t stream);

}  // namespace etc
