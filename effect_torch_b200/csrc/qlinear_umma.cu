// Dequant linear for prefill chunks and large batches (more than 128 vectors) on the 5th-generation tensor cores.
//
//   out[v, r] = sum_k x[v, k] * deq(W[r, k])        (quantized_linear, crates/runtime-cpu/src/quantized.rs:419-499)
//
// A CTA computes 256 weight rows x 128 vectors: two layout tiles of 128 rows, each the A operand of tcgen05.mma.kind::f16
// (M = 128, N = 128, K = 16) in TENSOR MEMORY, against one B operand of 128 vectors in shared memory ([K/8][128][8] f16, the
// canonical K-major layout, so that a stage of 128 columns is one contiguous bulk copy). Nineteen warps:
//   * weight loader / activation loader: bulk copies into rings of 3 to 6 and 3 stages, completion counted in bytes;
//   * sixteen dequant warps: a thread owns one TMEM lane = one weight row of one tile and half of a stage's blocks; it reads
//     16 or 32 payload bytes per block from shared memory, expands them to f16, scales and stores 16 TMEM columns;
//   * MMA warp: one elected lane issues 16 MMAs per stage (64 cycles each), tcgen05.commit frees TMEM slot and buffers.
// Tensor memory holds the two 128-column accumulators and two stages of the two expanded tiles.
//
// Why two row tiles x 128 vectors: a stage then moves 32 KB of activations and 18 KB of packed Q4_0 weights (from L2) for
// 1024 cycles of tensor work. One row tile x 256 vectors moved 64 KB + 9 KB, 69 bytes per cycle and SM, which is what L2 gave:
// 890 TFLOP/s on [14336 x 4096] x 512. Expansion takes half of the SM's issue slots and ends inside the MMAs of the stage
// before.
//
// Split-K over grid.z writes f32 partials that qlinear_reduce_kernel sums; with one split the epilogue (bias, residual add,
// SwiGLU over interleaved gate/up rows) runs straight from TMEM.
// Every mbarrier wait is bounded: on expiry the thread raises the abort flag and the status word, all roles fall through to
// the teardown, copies in flight are awaited, TMEM is freed and the kernel returns.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "activation.cuh"
#include "chain.cuh"
#include "codecs.cuh"
#include "dequant.cuh"
#include "kernels.h"

namespace etc {

namespace {

using namespace tc05;

constexpr int kUmmaRows = 128;    // of a layout tile
constexpr int kGemmTiles = 2;     // per CTA
constexpr int kGemmVectors = 128;
constexpr int kStageBlocks = 4;   // 32-value blocks per stage (K = 16 per MMA: 2 MMAs per block)
constexpr int kGemmDequantWarps = 16;
constexpr int kGemmWeightWarp = kGemmDequantWarps, kGemmMmaWarp = kGemmWeightWarp + 1, kGemmActivationWarp = kGemmMmaWarp + 1;
constexpr int kGemmThreads = (kGemmActivationWarp + 1) * 32;

template <int CODEC>
struct GemmCfg {
  static constexpr bool kNibbles = CODEC == 2 || CODEC == 12;
  static constexpr bool kPair = CODEC >= 12;  // two f16 per (row, block): (scale, min) or the two half-block scales
  static constexpr uint32_t kBlockQ = kNibbles ? 2048 : 4096;
  static constexpr uint32_t kBlockS = kPair ? 512 : 256;
  static constexpr uint32_t kTileQ = kStageBlocks * kBlockQ;
  static constexpr uint32_t kTileW = kStageBlocks * (kBlockQ + kBlockS);
  static constexpr uint32_t kStageW = kGemmTiles * kTileW;
  static constexpr uint32_t kStageB = kGemmVectors * kStageBlocks * 64;
  static constexpr int kSlots = 2;    // expanded stages in TMEM
  static constexpr int kStagesB = 3;
  static constexpr int kStagesW = kNibbles ? 6 : 3;
  static constexpr int kBars = 2 * kStagesW + 2 * kStagesB + kSlots + 1;
  static constexpr size_t kSmemBytes = (size_t)kStagesB * kStageB + (size_t)kStagesW * kStageW + kBars * sizeof(uint64_t) + 32;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");
};

struct GemmArgs {
  const unsigned char* quants;  // [tile][kblock][128 rows][16 B] or 8-bit codes [tile][kblock][128 rows][32 B]
  const unsigned char* scales;  // [tile][kblock][128] f16 or f16 pairs
  const __half* xh;             // [chunk][K/8][128][8] f16
  const float* bias;
  const float* residual;
  float* out;
  __half* out_xh;               // SwiGLU only: the result (also) as f16 for the next linear
  float* scratch;               // [chunk][split][128][rows_padded]
  unsigned long long* status;
  int vectors, rows, rows_padded, kblocks, epilogue;
  int tiles, tile0;             // of this launch (a segment of a weight fused from several codecs), and its first in the output
  int stages, stages_per_split;
};

template <int CODEC>
__global__ void __launch_bounds__(kGemmThreads, 1) qlinear_gemm_kernel(GemmArgs a) {
  using Cfg = GemmCfg<CODEC>;
  constexpr int WS = Cfg::kStagesW, BS = Cfg::kStagesB, AS = Cfg::kSlots, NV = kGemmVectors;
  constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(NV >> 3) << 17) | ((uint32_t)(kUmmaRows >> 4) << 24);  // f16 x f16 -> f32
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* b_ring = smem;
  unsigned char* w_ring = smem + BS * Cfg::kStageB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(w_ring + WS * Cfg::kStageW);
  // done[i % BS] completes when the MMAs of stage i have read its operands: it frees the activation buffer and the TMEM slot
  uint64_t *w_full = bars, *w_empty = w_full + WS, *b_full = w_empty + WS, *done = b_full + BS, *a_full = done + BS, *d_full = a_full + AS;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(d_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  chain_release();  // the next kernel of the stream may be scheduled already; it waits for this one
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int chunk = blockIdx.x, tile = blockIdx.y * kGemmTiles, split = blockIdx.z;
  const int live_tiles = min(kGemmTiles, a.tiles - tile);
  const int s0 = split * a.stages_per_split, n = min(a.stages, s0 + a.stages_per_split) - s0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < WS; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], kGemmDequantWarps); }
    for (int i = 0; i < BS; ++i) { mbar_init(&b_full[i], 1); mbar_init(&done[i], 1); }
    for (int i = 0; i < AS; ++i) mbar_init(&a_full[i], kGemmDequantWarps);
    mbar_init(d_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kGemmMmaWarp) tmem_alloc(tmem_holder, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;  // accumulator of tile t at columns [t * NV, (t + 1) * NV), then the expanded stages
  const uint32_t a_tmem = tmem + kGemmTiles * NV;

  if (warp < kGemmDequantWarps) {
    // ------------------------------------------------------------------ dequant warps
    const int mine = (warp >> 2) & 1, half = warp >> 3, row = (warp & 3) * 32 + lane;  // tile, half of the stage's blocks, row
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const unsigned char* payload = w_ring + mine * Cfg::kTileW + row * (Cfg::kBlockQ / kUmmaRows);
    const unsigned char* scales = w_ring + mine * Cfg::kTileW + Cfg::kTileQ + row * (Cfg::kBlockS / kUmmaRows);
    {
      Ring<WS> w;
      Ring<AS> slot;
      Ring<BS> freed;  // the stage AS before this one
      bool ok = true;
      for (int i = 0; i < n && ok; ++i) {
        ok = wait_warp(&w_full[w.at], w.parity, abort_flag) && (i < AS || wait_warp(&done[freed.at], freed.parity, abort_flag));
        if (!ok) break;
        if (i >= AS) freed.next();
        tc_fence_after();
        if (mine < live_tiles) {
          const uint32_t stage = (uint32_t)w.at * Cfg::kStageW;
          constexpr int kMine = kStageBlocks / 2;  // blocks beyond the weight's K hold stale bytes that no MMA reads
          const unsigned char* q = payload + stage + half * kMine * Cfg::kBlockQ;
          const uint32_t cols = a_tmem + lane_base + (uint32_t)((slot.at * kGemmTiles + mine) * kStageBlocks * 16 + half * kMine * 16);
          uint32_t first[kMine], second[kMine];
#pragma unroll
          for (int b = 0; b < kMine; ++b) load_scales<CODEC>(scales + stage + (half * kMine + b) * Cfg::kBlockS, first[b], second[b]);
          auto expand = [&](auto large) {
#pragma unroll
            for (int b = 0; b < kMine; ++b) {
              uint32_t regs[16];
              expand_block<CODEC, decltype(large)::value>(q + b * Cfg::kBlockQ, first[b], second[b], regs);
              tmem_st16(cols + b * 16, regs);
            }
          };
          if (small_scales<CODEC>(first, second)) expand(std::false_type());
          else expand(std::true_type());
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_empty[w.at]);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[slot.at]);
        w.next();
        slot.next();
      }
    }
    // ------------------------------------------------------------------ epilogue: half of a tile's vectors per warp
    chain_wait();  // outputs, residual and scratch may still be in use by the kernel before this one
    if (wait_warp(d_full, 0, abort_flag) && mine < live_tiles) {
      tc_fence_after();
      const int r = (a.tile0 + tile + mine) * kUmmaRows + row;
      const int v_base = chunk * NV;
      const float bias_v = a.bias && r < a.rows ? a.bias[r] : 0.0f;
      const bool partial = gridDim.z > 1;
#pragma unroll 1
      for (int v0 = half * (NV / 2); v0 < (half + 1) * (NV / 2) && v_base + v0 < a.vectors; v0 += 16) {
        uint32_t bits[16];
        tmem_ld16(tmem + lane_base + (uint32_t)(mine * NV + v0), bits);
        tmem_wait_ld();
        const int left = a.vectors - v_base - v0;
        if (partial) {
          float* dst = a.scratch + (((size_t)chunk * gridDim.z + split) * NV + v0) * a.rows_padded + r;
#pragma unroll
          for (int v = 0; v < 16; ++v) dst[(size_t)v * a.rows_padded] = __uint_as_float(bits[v]);
        } else if (a.epilogue == ETC_EPILOGUE_SWIGLU) {
          // rows are interleaved in groups of 8: lanes 0-7 of each 16 hold gate rows, lanes 8-15 their up rows; of two
          // vectors the gate lane finishes the first and the up lane the second
          const bool is_up = r & 8;
          const int oc = (r >> 4) * 8 + (r & 7);
#pragma unroll
          for (int v = 0; v < 16; v += 2) {
            const float first = __uint_as_float(bits[v]) + bias_v, second = __uint_as_float(bits[v + 1]) + bias_v;
            const float other = __shfl_xor_sync(0xffffffffu, is_up ? first : second, 8);
            const float act = silu_tanh(is_up ? other : first) * (is_up ? second : other);
            const int at = v_base + v0 + v + is_up;
            if (oc >= a.rows / 2 || v + is_up >= left) continue;
            if (a.out) a.out[(size_t)at * (a.rows / 2) + oc] = act;
            if (a.out_xh) a.out_xh[hand_off_cell(oc >> 3, at, NV, a.rows / 16) + (oc & 7)] = half_sat(act);
          }
        } else if (r < a.rows) {
          const size_t at = (size_t)(v_base + v0) * a.rows + r;
          float extra[16];
#pragma unroll
          for (int v = 0; v < 16; ++v) extra[v] = a.epilogue == ETC_EPILOGUE_RESIDUAL && v < left ? a.residual[at + (size_t)v * a.rows] : 0.0f;
#pragma unroll
          for (int v = 0; v < 16; ++v)
            if (v < left) a.out[at + (size_t)v * a.rows] = extra[v] + (__uint_as_float(bits[v]) + bias_v);
        }
      }
    }
  } else if (warp == kGemmWeightWarp) {
    // ------------------------------------------------------------------ weight loader (one lane)
    if (elect_one()) {
      Ring<WS> w;
      int issued = 0;
      for (int i = 0; i < n; ++i) {
        if (!mbar_wait(&w_empty[w.at], w.parity ^ 1u, abort_flag)) break;
        const int kb = (s0 + i) * kStageBlocks;
        const uint32_t valid = (uint32_t)min(kStageBlocks, a.kblocks - kb);
        unsigned char* dst = w_ring + (size_t)w.at * Cfg::kStageW;
        mbar_arrive_expect_tx(&w_full[w.at], (uint32_t)live_tiles * valid * (Cfg::kBlockQ + Cfg::kBlockS));
        for (int t = 0; t < live_tiles; ++t) {
          const size_t block = (size_t)(tile + t) * a.kblocks + kb;
          bulk_copy_g2s(dst + t * Cfg::kTileW, a.quants + block * Cfg::kBlockQ, valid * Cfg::kBlockQ, &w_full[w.at]);
          bulk_copy_g2s(dst + t * Cfg::kTileW + Cfg::kTileQ, a.scales + block * Cfg::kBlockS, valid * Cfg::kBlockS, &w_full[w.at]);
        }
        issued = i + 1;
        w.next();
      }
      if (*abort_flag)  // give up: this warp's own copies land (bounded) before shared memory is released
        for (int i = max(0, issued - WS); i < issued; ++i)
          for (unsigned spin = 0; spin < (1u << 20) && !mbar_try_wait(&w_full[i % WS], (uint32_t)(i / WS) & 1u); ++spin) __nanosleep(64);
    }
  } else if (warp == kGemmActivationWarp) {
    // ------------------------------------------------------------------ activation loader (one lane)
    if (elect_one()) {
      chain_wait();  // the activations come from the kernel before this one
      const __half* xh = a.xh + (size_t)chunk * a.kblocks * 4 * NV * 8;
      Ring<BS> b;
      int issued = 0;
      for (int i = 0; i < n; ++i) {
        if (i >= BS && !mbar_wait(&done[b.at], b.parity ^ 1u, abort_flag)) break;  // stage i - BS used this buffer and barrier
        const int kb = (s0 + i) * kStageBlocks;
        const uint32_t bytes = (uint32_t)min(kStageBlocks, a.kblocks - kb) * 4u * NV * 16u;
        mbar_arrive_expect_tx(&b_full[b.at], bytes);
        bulk_copy_g2s(b_ring + (size_t)b.at * Cfg::kStageB, xh + (size_t)kb * 4 * NV * 8, bytes, &b_full[b.at]);
        issued = i + 1;
        b.next();
      }
      if (*abort_flag)
        for (int i = max(0, issued - BS); i < issued; ++i)
          for (unsigned spin = 0; spin < (1u << 20) && !mbar_try_wait(&b_full[i % BS], (uint32_t)(i / BS) & 1u); ++spin) __nanosleep(64);
    }
  } else {
    // ------------------------------------------------------------------ MMA issuer (one lane)
    if (elect_one()) {
      Ring<BS> b;
      Ring<AS> slot;
      bool ok = true;
      const uint64_t desc0 = make_b_desc(smem_u32(b_ring), NV * 16u, 128u);
      for (int i = 0; i < n && ok; ++i) {
        ok = mbar_wait(&b_full[b.at], b.parity, abort_flag) && mbar_wait(&a_full[slot.at], slot.parity, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const int valid = min(kStageBlocks, a.kblocks - (s0 + i) * kStageBlocks);
        // two K = 16 instructions per block and tile: two column groups of B, 8 TMEM columns of A each; whole stages unrolled
        // with constant steps, so that the operands stay in uniform registers
        const uint64_t desc = desc0 + (uint64_t)(b.at * (int)(Cfg::kStageB / 16));
        const uint32_t a0 = a_tmem + (uint32_t)(slot.at * kGemmTiles * kStageBlocks * 16), a1 = a0 + kStageBlocks * 16;
        umma_ts(tmem, a0, desc, kIdesc, i > 0 ? 1u : 0u);
        umma_ts(tmem + NV, a1, desc, kIdesc, i > 0 ? 1u : 0u);
        if (valid == kStageBlocks) {
#pragma unroll
          for (int j = 1; j < 2 * kStageBlocks; ++j) {
            umma_ts(tmem, a0 + 8u * j, desc + 2u * NV * j, kIdesc, 1u);
            umma_ts(tmem + NV, a1 + 8u * j, desc + 2u * NV * j, kIdesc, 1u);
          }
        } else {
          for (int j = 1; j < 2 * valid; ++j) {
            umma_ts(tmem, a0 + 8u * j, desc + 2u * NV * j, kIdesc, 1u);
            umma_ts(tmem + NV, a1 + 8u * j, desc + 2u * NV * j, kIdesc, 1u);
          }
        }
        tc_commit(&done[b.at]);
        b.next();
        slot.next();
      }
      if (ok) tc_commit(d_full);
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(a.status, 0ull, 3ull);  // bounded wait expired
  if (warp == kGemmMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Repack raw GGUF rows into the per-thread streaming layout: for row tile t and block kb the 128 rows'
// 16 (Q4_0) or 32 (Q8_0) payload bytes are contiguous, so each warp load instruction is 512 contiguous bytes.
__global__ void repack_umma_kernel(RepackParts parts, int codec, int64_t rows, int64_t rows_padded, int64_t kblocks,
                                   int interleave8, uint32_t* __restrict__ quants, __half* __restrict__ scales) {
  const int64_t total = rows_padded * kblocks;
  const bool kquant = codec >= 11;
  const int bb = codec == 2 ? 18 : (codec == 8 ? 34 : (codec == 11 ? 110 : (codec == 12 ? 144 : (codec == 13 ? 176 : 210))));  // bytes per source block
  const int per_block = kquant ? 8 : 1;                                              // 32-value blocks per source block
  const int words = (codec == 2 || codec == 12) ? 4 : 8;
  const int64_t row_bytes = kblocks / per_block * bb;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / kblocks, kb = idx - r * kblocks;
    const uint8_t* src_row = nullptr;
    if (r < rows) {
      if (interleave8) {
        const int64_t grp = r >> 4, within = r & 15;
        src_row = parts.ptr[within >= 8 ? 1 : 0] + (grp * 8 + (within & 7)) * row_bytes;
      } else {
        int64_t rr = r;
        for (int p = 0; p < parts.n_parts; ++p) {
          if (rr < parts.rows[p]) { src_row = parts.ptr[p] + rr * row_bytes; break; }
          rr -= parts.rows[p];
        }
      }
    }
    const int64_t tile = r / kUmmaRows, row = r % kUmmaRows;
    uint32_t* dst = quants + ((tile * kblocks + kb) * kUmmaRows + row) * words;
    __half scale = __float2half_rn(0.0f), second = __float2half_rn(0.0f);
    const int pos[8] = {0, 16, 8, 24, 4, 20, 12, 28}, byte_pos[4] = {0, 16, 8, 24};
    // the positions that dequant.cuh reads: every word three bits up, signed bytes plus 128
    auto place = [](uint32_t word) { return __funnelshift_l(word, word, 3); };
    if (!src_row) {
      for (int w = 0; w < words; ++w) dst[w] = 0u;  // the scales are 0
    } else if (codec == 12) {
      // Q4_K (crates/runtime-cpu/src/quantized.rs:180-199): sub-block `sub` of the 256-value block, value = d*sc*code - dmin*m
      const uint8_t* blk = src_row + (kb >> 3) * bb;
      const int sub = (int)(kb & 7);
      int sc, mn;
      scale_min_k4(sub, blk + 4, sc, mn);
      scale = __float2half_rn(__fmul_rn(fp16_at(blk, 0), (float)sc));
      second = __float2half_rn(__fmul_rn(fp16_at(blk, 2), (float)mn));
      for (int w = 0; w < 4; ++w) {
        uint32_t word = 0;
        for (int j = 0; j < 8; ++j) {
          const int raw = blk[16 + (sub >> 1) * 32 + 8 * w + j];
          word |= (uint32_t)((sub & 1) ? (raw >> 4) : (raw & 0x0f)) << pos[j];
        }
        dst[w] = place(word);
      }
    } else if (codec == 11) {
      // Q3_K (quantized.rs:142-176): block `sub` of the 256-value block is groups 2*sub and 2*sub+1 of 16 values,
      // value = d*(scale6 - 32)*(low2 - (high bit clear ? 4 : 0)); stored as byte codes (plus 128) with one f16 scale per
      // group, the layout of the re-cut Q6_K
      const uint8_t* blk = src_row + (kb >> 3) * bb;
      const int sub = (int)(kb & 7), half = sub >> 2, lane = sub & 3;
      const uint8_t* packed = blk + 96;
      const float d = fp16_at(blk, 108);
      auto group_scale = [&](int g) {
        const int low = g < 8 ? (packed[g] & 0x0f) : (packed[g - 8] >> 4);
        const int high = (packed[8 + g % 4] >> (2 * (g / 4))) & 3;
        return __float2half_rn(__fmul_rn(d, (float)((low | (high << 4)) - 32)));
      };
      scale = group_scale(2 * sub);
      second = group_scale(2 * sub + 1);
      const uint8_t mask = (uint8_t)(1u << (half * 4 + lane));
      for (int w = 0; w < 8; ++w) {
        uint32_t word = 0;
        for (int j = 0; j < 4; ++j) {
          const int v = 4 * w + j;
          const int code = ((blk[32 + half * 32 + v] >> (2 * lane)) & 3) - ((blk[v] & mask) == 0 ? 4 : 0);
          word |= (uint32_t)(code + 128) << byte_pos[j];
        }
        dst[w] = place(word);
      }
    } else if (codec == 13) {
      // Q5_K (quantized.rs:203-234): sub-block `sub`, value = d*sc*code - dmin*m with a 5-bit code (low nibble + one high
      // bit); stored as int8 codes with (scale, min) per 32 values
      const uint8_t* blk = src_row + (kb >> 3) * bb;
      const int sub = (int)(kb & 7);
      int sc, mn;
      scale_min_k4(sub, blk + 4, sc, mn);
      scale = __float2half_rn(__fmul_rn(fp16_at(blk, 0), (float)sc));
      second = __float2half_rn(__fmul_rn(fp16_at(blk, 2), (float)mn));
      const uint8_t* ql = blk + 48 + (sub >> 1) * 32;
      const uint8_t mask = (uint8_t)(1u << sub);
      for (int w = 0; w < 8; ++w) {
        uint32_t word = 0;
        for (int j = 0; j < 4; ++j) {
          const int v = 4 * w + j;
          const int code = ((sub & 1) ? (ql[v] >> 4) : (ql[v] & 0x0f)) + ((blk[16 + v] & mask) == 0 ? 0 : 16);
          word |= (uint32_t)code << byte_pos[j];
        }
        dst[w] = place(word);
      }
    } else if (codec == 14) {
      // Q6_K (quantized.rs:238-261): values 32*sub .. 32*sub+31 of the 256-value block, value = d*scale*(code - 32) with one
      // int8 scale per 16 values
      const uint8_t* blk = src_row + (kb >> 3) * bb;
      const int first = (int)(kb & 7) * 32;
      const int half = first >> 7, quarter = (first & 127) >> 5;
      const uint8_t* ql = blk + half * 64;
      const uint8_t* qh = blk + 128 + half * 32;
      const float d = fp16_at(blk, 208);
      scale = __float2half_rn(__fmul_rn(d, (float)(int)(signed char)blk[192 + half * 8 + quarter * 2]));
      second = __float2half_rn(__fmul_rn(d, (float)(int)(signed char)blk[192 + half * 8 + quarter * 2 + 1]));
      for (int w = 0; w < 8; ++w) {
        uint32_t word = 0;
        for (int j = 0; j < 4; ++j) {
          const int index = 4 * w + j;
          const int low = (quarter & 1) ? ql[index + 32] : ql[index];
          const int low4 = (quarter & 2) ? (low >> 4) : (low & 0x0f);
          const int code = (low4 | (((qh[index] >> (2 * quarter)) & 3) << 4)) - 32;
          word |= (uint32_t)(code + 128) << byte_pos[j];
        }
        dst[w] = place(word);
      }
    } else {
      const uint8_t* blk = src_row + kb * bb;
      scale = __ushort_as_half((unsigned short)(blk[0] | (blk[1] << 8)));
      if (codec == 2) {
        for (int w = 0; w < 4; ++w) {
          uint32_t word = 0;
          for (int j = 0; j < 8; ++j) {
            const int i = 8 * w + j;
            const uint32_t code = i < 16 ? (blk[2 + i] & 0x0fu) : (uint32_t)(blk[2 + i - 16] >> 4);
            word |= code << pos[j];
          }
          dst[w] = place(word);
        }
      } else {
        for (int w = 0; w < 8; ++w) {
          uint32_t word = 0;
          for (int j = 0; j < 4; ++j) word |= (uint32_t)(blk[2 + 4 * w + j] ^ 0x80u) << byte_pos[j];
          dst[w] = place(word);
        }
      }
    }
    if (kquant) {
      scales[((tile * kblocks + kb) * kUmmaRows + row) * 2] = scale;
      scales[((tile * kblocks + kb) * kUmmaRows + row) * 2 + 1] = second;
    } else {
      scales[(tile * kblocks + kb) * kUmmaRows + row] = scale;
    }
  }
}

template <int CODEC>
cudaError_t launch_gemm_pass(const GemmArgs& args, int chunks, int splits, cudaStream_t stream) {
  constexpr size_t smem = GemmCfg<CODEC>::kSmemBytes;
  auto kernel = qlinear_gemm_kernel<CODEC>;
  const cudaError_t attr = opt_in_shared_memory(kernel, smem);
  if (attr != cudaSuccess) return attr;
  // chained: set-up and the first weight stages do not depend on the previous kernel and start under its tail
  return launch_chained(kernel, dim3((unsigned)chunks, (unsigned)((args.tiles + kGemmTiles - 1) / kGemmTiles), (unsigned)splits), dim3(kGemmThreads), smem, stream, args);
}

}  // namespace

cudaError_t launch_repack(const TiledWeight& w, const RepackParts& parts, cudaStream_t stream) {
  const int64_t kblocks = w.columns / 32;
  const int64_t total = w.rows_padded * kblocks;
  if (total == 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 32);
  repack_umma_kernel<<<grid, 256, 0, stream>>>(parts, w.codec, w.rows, w.rows_padded, kblocks, w.interleave8, (uint32_t*)w.quants, w.scales);
  return cudaGetLastError();
}

UmmaPlan plan_umma(const TiledWeight& w, int64_t vectors, int sm_count) {
  UmmaPlan p;
  p.chunks = (int)std::max<int64_t>(1, (vectors + p.nv - 1) / p.nv);
  p.tiles = (int)(w.rows_padded / kUmmaRows);
  p.stages = (int)((w.columns / 32 + kStageBlocks - 1) / kStageBlocks);
  // as many splits as there are SMs for (one CTA each), of at least two stages
  const int ctas = (p.tiles + kGemmTiles - 1) / kGemmTiles * p.chunks;
  const int splits = std::min(std::max(1, std::max(1, sm_count) / ctas), std::max(1, p.stages / 2));
  p.stages_per_split = (p.stages + splits - 1) / splits;
  p.splits = (p.stages + p.stages_per_split - 1) / p.stages_per_split;
  p.xh_bytes = (size_t)p.chunks * (w.columns / 8) * p.nv * 16;
  p.scratch_bytes = p.splits > 1 ? (size_t)p.chunks * p.splits * p.nv * w.rows_padded * sizeof(float) : 0;
  return p;
}

// qlinear_reduce_kernel lives in quant_kernels.cu
cudaError_t launch_qlinear_umma(const TiledWeight& w, const float* x, const __half* xh_ready, int64_t vectors, const float* bias,
                                const float* residual, int epilogue, float* out, __half* out_xh, __half* xh, float* scratch, DeviceStatus* status, int sm_count, cudaStream_t stream,
                                int* launches) {
  if (vectors <= 0) return cudaSuccess;
  const UmmaPlan plan = plan_umma(w, vectors, sm_count);
  const int K = (int)w.columns;
  cudaError_t e = cudaSuccess;
  if (!xh_ready) {
    e = launch_hand_off_convert(x, vectors, K, plan.nv, xh, sm_count, stream);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  GemmArgs args;
  args.xh = xh_ready ? xh_ready : xh;
  args.out_xh = epilogue == ETC_EPILOGUE_SWIGLU ? out_xh : nullptr;
  args.bias = bias;
  args.residual = residual;
  args.out = out;
  args.scratch = scratch;
  args.status = &status->code;
  args.vectors = (int)vectors;
  args.rows = (int)w.rows;
  args.rows_padded = (int)w.rows_padded;
  args.kblocks = K / 32;
  args.epilogue = epilogue;
  args.stages = plan.stages;
  args.stages_per_split = plan.stages_per_split;
  // one launch per run of equal codecs; all of them share the plan (split count, partial layout) of the whole weight
  for (int sgm = 0; sgm < std::max(1, w.n_segments); ++sgm) {
    int codec = w.codec;
    args.quants = w.quants;
    args.scales = reinterpret_cast<const unsigned char*>(w.scales);
    args.tiles = plan.tiles;
    args.tile0 = 0;
    if (w.n_segments > 0) {
      const TiledSegment& seg = w.segments[sgm];
      codec = seg.codec;
      args.tiles = seg.tiles;
      args.tile0 = seg.tile0;
      args.quants += seg.quant_offset;
      args.scales += seg.scale_offset;
    }
    switch (codec) {
      case 2: e = launch_gemm_pass<2>(args, plan.chunks, plan.splits, stream); break;
      case 8: e = launch_gemm_pass<8>(args, plan.chunks, plan.splits, stream); break;
      case 12: e = launch_gemm_pass<12>(args, plan.chunks, plan.splits, stream); break;
      case 13: e = launch_gemm_pass<13>(args, plan.chunks, plan.splits, stream); break;
      default: e = launch_gemm_pass<14>(args, plan.chunks, plan.splits, stream);  // 14, and 11 whose re-cut form is the same
    }
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  if (plan.splits == 1) return cudaSuccess;
  if (launches) ++*launches;
  return launch_qlinear_reduce(scratch, plan.splits, plan.nv, (int)vectors, (int)w.rows, (int)w.rows_padded, bias, residual, epilogue, out, args.out_xh, plan.nv, stream);
}

}  // namespace etc
