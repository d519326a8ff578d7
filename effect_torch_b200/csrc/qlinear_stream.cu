// Dequant linear for decode batches (up to 128 vectors) on the 5th-generation tensor cores, streaming weights at HBM rate.
//
//   out[v, r] = sum_k x[v, k] * deq(W[r, k])        (quantized_linear, crates/runtime-cpu/src/quantized.rs:419-499)
//
// The 128 rows of a layout tile are the A operand of tcgen05.mma.kind::f16 (M = 128, N = NV, K = 16) in tensor memory; the
// NV input vectors are the B operand in shared memory, in the canonical K-major layout the producer already stored
// ([K/8][NV][8] f16). A CTA does one tile, or a range of its K, with eleven warps:
//   * weight loader: bulk copies (cp.async.bulk, completion counted in bytes on an mbarrier) of the packed weights and block
//     scales of a stage (128 rows x 128 columns) into a deep shared-memory ring. Weights depend on no earlier kernel, so
//     under programmatic dependent launch the whole ring is requested while the previous kernel still runs.
//   * activation loader: the stage's B operand, one bulk copy, after the grid dependency wait.
//   * two groups of four dequant warps (stages alternate): a thread owns one TMEM lane = one weight row, reads 16 payload
//     bytes per 32-value block from the ring, expands to f16, scales and stores 16 TMEM columns per block.
//   * MMA warp: one elected lane issues 8 MMAs per stage (N / 2 cycles each); tcgen05.commit frees the stage's buffers.
// Two CTAs share an SM (half the shared memory, 256 TMEM columns each), so that one expands while the other starts, waits
// or stores; a CTA of the next launch can take the place of one that has ended and fill its ring under this launch's tail.
//
// Split over K. Deferred sums: grid (splits, tiles), partial sums to memory, added up by the kernel that consumes them.
// Otherwise the CTAs of a tile form a cluster: each puts its accumulator into its shared memory, and after a cluster
// barrier every CTA adds up, in rank order, its share of the vectors from all of them and runs the epilogue. (Equal runs
// of (tile, stage) units with the pieces of cut tiles exchanged through memory and a ticket per tile took 10 to 17 us for
// the exchange on [28672 x 4096] and [4096 x 4096]: a fence, an atomic and a chain of L2 round trips.)
//
// Roofline: HBM, rows*K/32*{18,34} bytes. A dequant warp has 255 instructions per stage of 128 x 128 Q4_0 weights (an FMA
// and a mask per pair, see dequant.cuh); with the loaders and the MMA warp an SM issues 1306 per stage, at 65 % of its slots.
// [128256 x 4096] x 32, activations ready, with the codes spliced and scaled in two steps and as it is: 547 and 506 cycles per
// stage (HBM delivers one in 410), 79.1 and 73.3 us; x 64: 90.4 and 85.8; [28672 x 4096] x 32: 26.5 and 24.1. In the form for
// up to 16 vectors: Q4_0 [128256 x 4096] v8 70.5 us, Q8_0 100.4 (0.88 of the copy bandwidth). The rest is the start of a
// launch (3 us to the first MMA), the uneven last tiles and the epilogue.
//
// Every mbarrier wait is bounded: on expiry the abort flag and the status word (3) are raised, all roles run dry, copies
// in flight are awaited, TMEM is freed.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "activation.cuh"
#include "chain.cuh"
#include "dequant.cuh"
#include "kernels.h"

namespace etc {

namespace {

namespace cg = cooperative_groups;
using namespace tc05;

constexpr int kRows = 128;       // of a layout tile
constexpr int kStageBlocks = 4;  // 32-value blocks per stage
constexpr int kDequantGroups = 2;
constexpr int kWeightWarp = 4 * kDequantGroups, kMmaWarp = kWeightWarp + 1, kActivationWarp = kMmaWarp + 1;
constexpr int kMaxStreamCluster = 8;  // the portable size
constexpr int kStreamThreads = (kActivationWarp + 1) * 32;

constexpr int kExactVectors = 16;
constexpr int kDirectVectors = 4;  // at most these many f32 vectors are converted by the linear itself

template <int CODEC, int NV>
struct StreamCfg {
  static constexpr bool kNibbles = CODEC == 2 || CODEC == 12;
  static constexpr bool kPair = CODEC >= 12;  // two f16 per (row, block): (scale, min) or the two half-block scales
  static constexpr uint32_t kBlockQ = kNibbles ? 2048 : 4096;
  static constexpr uint32_t kBlockS = kPair ? 512 : 256;
  static constexpr uint32_t kStageQ = kStageBlocks * kBlockQ;
  static constexpr uint32_t kStageW = kStageBlocks * (kBlockQ + kBlockS);
  static constexpr uint32_t kStageB = NV * kStageBlocks * 64;
  // Up to 16 vectors, Q4_0 and Q8_0: the codes go through the MMA unscaled and every block has an accumulator of its own,
  // whose sums the dequant warps multiply by the block's f32 scale (16 FMA per row in place of 16 products on f16 pairs).
  static constexpr bool kExact = NV == kExactVectors;
  static constexpr int kSlots = NV == 32 ? 3 : 2;  // expanded stages in TMEM
  static constexpr int kAccumulators = kExact ? kSlots * kStageBlocks : 1;
  static constexpr int kStagesB = NV <= 32 ? (kNibbles || kExact ? 6 : 4) : (NV <= 64 && kNibbles ? 3 : 2);
  // a whole number of stages per dequant group: a ring buffer then belongs to one group, whose own previous round is what
  // tells two phases of the buffer's barrier apart (copies of neighbouring stages may land in either order)
  static constexpr int kStagesW = (int)((104u * 1024 - kStagesB * kStageB) / kStageW) / kDequantGroups * kDequantGroups;
  static constexpr uint32_t kTmemCols = 256;
  static constexpr int kDone = kStagesB > kSlots ? kStagesB : kSlots;  // barriers on which the MMAs of a stage report
  static constexpr int kBars = 2 * kStagesW + kStagesB + kSlots + kDone + 1;
  static constexpr size_t kSmemBytes = (size_t)kStagesB * kStageB + (size_t)kStagesW * kStageW + kBars * sizeof(uint64_t) + 32;
  static_assert(NV * kAccumulators + kSlots * kStageBlocks * 16 <= (int)kTmemCols, "tensor memory of half an SM");
  static_assert(kStagesW >= kDequantGroups, "ring");
  static_assert(kSmemBytes <= 112 * 1024, "two CTAs per SM");
  static_assert((size_t)NV * kRows * sizeof(float) <= (size_t)kStagesB * kStageB + (size_t)kStagesW * kStageW, "the accumulator fits the rings");
};

struct StreamArgs {
  const unsigned char* quants;  // [tile][kblock][128 rows][16 B] or 8-bit codes [tile][kblock][128 rows][32 B]
  const unsigned char* scales;  // [tile][kblock][128] f16 or f16 pairs
  const __half* xh;             // [K/8][xh_nv][8] f16; xh_nv == NV but for the exact form, where it may be wider
  const float* x;               // exact form without xh: f32 [vectors, K]
  int xh_nv;
  const float* bias;
  const float* residual;
  float* out;
  float* scratch;               // deferred sums: [splits][NV][rows_padded]
  unsigned long long* status;
  __half* out_xh;               // optional: the result also as f16 [cols/8][out_xh_nv][8] for the next linear
  int out_xh_nv;
  int vectors, rows, rows_padded, kblocks, epilogue;
  int tile0;                    // first tile of this launch in the output (a segment of a weight fused from several codecs)
  int stages, stages_per_split; // of a tile; of a CTA
  int deferred;                 // partial sums only
};

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Four consecutive values of an output row: columns c .. c + 3 of vector v, the first `n` of them inside the row.
__device__ __forceinline__ void store4(const StreamArgs& a, int v, int c, int n, int out_cols, const float4& val) {
  if (a.out) {
    float* dst = a.out + (size_t)v * out_cols + c;
    if (n == 4 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
      *reinterpret_cast<float4*>(dst) = val;
    } else {
      dst[0] = val.x;
      if (n > 1) dst[1] = val.y;
      if (n > 2) dst[2] = val.z;
      if (n > 3) dst[3] = val.w;
    }
  }
  if (a.out_xh) *reinterpret_cast<uint2*>(a.out_xh + ((size_t)(c >> 3) * a.out_xh_nv + v) * 8 + (c & 7)) = pack4(val);
}

__device__ __forceinline__ void dequant_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(4 * kDequantGroups * 32) : "memory"); }

template <int CODEC, int NV, int USED = NV>
__global__ void __launch_bounds__(kStreamThreads, 2) qlinear_stream_kernel(StreamArgs a) {
  using Cfg = StreamCfg<CODEC, NV>;
  constexpr int WS = Cfg::kStagesW, BS = Cfg::kStagesB, AS = Cfg::kSlots, DONE = Cfg::kDone;
  constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(NV >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);  // f16 x f16 -> f32
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* b_ring = smem;
  unsigned char* w_ring = smem + BS * Cfg::kStageB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(w_ring + WS * Cfg::kStageW);
  // `done[i % DONE]` completes when the MMAs of stage i have read its operands: one commit frees both the TMEM slot and the
  // activation buffer, whose owners wait for the stage that used them last (at most DONE stages back)
  uint64_t *w_full = bars, *w_empty = w_full + WS, *b_full = w_empty + WS, *a_full = b_full + BS;
  uint64_t *done = a_full + AS, *d_full = done + DONE;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(d_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  chain_release();  // the next kernel of the stream may be scheduled already; it waits for this one
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int split = blockIdx.x, tile = blockIdx.y;
  const int s0 = split * a.stages_per_split, n = min(a.stages, s0 + a.stages_per_split) - s0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < WS; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 4); }
    for (int i = 0; i < BS; ++i) mbar_init(&b_full[i], 1);
    for (int i = 0; i < AS; ++i) mbar_init(&a_full[i], 4);
    for (int i = 0; i < DONE; ++i) mbar_init(&done[i], 1);
    mbar_init(d_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tmem_alloc(tmem_holder, Cfg::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;         // the accumulators from column 0, then the expanded stages
  const uint32_t a_tmem = tmem + NV * Cfg::kAccumulators;

  if (warp < kWeightWarp) {
    // ------------------------------------------------------------------ dequant warps
    const int group = warp >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    Ring<WS> w;
    Ring<AS> slot;
    Ring<DONE> freed;  // the stage AS before this one
    w.skip(group);
    slot.skip(group);
    int behind = group - AS;
    const unsigned char* payload = w_ring + row * (Cfg::kBlockQ / kRows);
    const unsigned char* scales = w_ring + Cfg::kStageQ + row * (Cfg::kBlockS / kRows);
    bool ok = true;
    // exact form: the first USED sums of this row, and the block scales of the stage whose products are not added yet
    float sums[Cfg::kExact ? USED : 1], scale[kStageBlocks], next_scale[kStageBlocks];
#pragma unroll
    for (int v = 0; v < (Cfg::kExact ? USED : 1); ++v) sums[v] = 0.0f;
    auto load_products = [&](uint32_t taddr, auto& products) {
      if constexpr (USED == 8) tmem_ld8(taddr, products);
      else tmem_ld16(taddr, products);
    };
    auto add_block = [&](auto& products, float block_scale) {
      pin(products);
#pragma unroll
      for (int v = 0; v < (Cfg::kExact ? USED : 0); ++v) sums[v] = fmaf(block_scale, __uint_as_float(products[v]), sums[v]);
    };
    constexpr int GROUP = 16 / USED;  // blocks whose products are in registers at a time (all that there is room for)
    const uint32_t my_products = tmem + lane_base + (uint32_t)(group * kStageBlocks * NV);
    for (int i = group; i < n && ok; i += kDequantGroups) {
      ok = wait_warp(&w_full[w.at], w.parity, abort_flag);
      if (!ok) break;
      const uint32_t stage = (uint32_t)w.at * Cfg::kStageW;
      int hands_back = 0;  // the lane that arrives on w_empty
      auto slot_is_free = [&] {
        ok = behind < 0 || wait_warp(&done[freed.at], freed.parity, abort_flag);
        if (ok) tc_fence_after();
        return ok;
      };
      const uint32_t slot_cols = a_tmem + lane_base + (uint32_t)(slot.at * kStageBlocks * 16);
      if constexpr (Cfg::kExact) {
        if (!slot_is_free()) break;
        // the products of the stage AS before this one (a whole one), whose slot and accumulators this one takes over
        uint32_t products[GROUP][USED];
        uint32_t seen = 0;
#pragma unroll
        for (int b = 0; b < kStageBlocks; ++b) {  // blocks beyond the tile's K hold stale bytes that no MMA reads
          uint32_t regs[16];
          if (behind >= 0 && b % GROUP == 0) {
#pragma unroll
            for (int j = 0; j < GROUP; ++j) load_products(my_products + (uint32_t)((b + j) * NV), products[j]);
          }
          expand_codes<CODEC>(payload + stage + b * Cfg::kBlockQ, regs);
          const uint32_t bits = *reinterpret_cast<const unsigned short*>(scales + stage + b * Cfg::kBlockS);
          seen ^= bits;
          next_scale[b] = __half2float(__ushort_as_half((unsigned short)bits)) * kCodeUnits;
          tmem_st16(slot_cols + b * 16, regs);
          if (behind >= 0 && b % GROUP == GROUP - 1) {
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < GROUP; ++j) add_block(products[j], scale[b - GROUP + 1 + j]);
          }
        }
#pragma unroll
        for (int b = 0; b < kStageBlocks; ++b) scale[b] = next_scale[b];
        // The scales are used a round later. An arrival on w_empty does not wait for loads whose results nothing has used yet
        // (nor does a fence): the next round's bytes came back as scales, in one step of some fifty where launches overlap
        // just so. Which of two lanes arrives therefore hangs on a bit of every scale that the warp has loaded: the vote has
        // no result before all of them are in registers, whatever order the instructions are put in.
        hands_back = __popc(__ballot_sync(0xffffffffu, seen & 1u)) & 1;
      } else {
        uint32_t first[kStageBlocks], second[kStageBlocks];
#pragma unroll
        for (int b = 0; b < kStageBlocks; ++b) load_scales<CODEC>(scales + stage + b * Cfg::kBlockS, first[b], second[b]);
        auto expand = [&](auto large) {
#pragma unroll
          for (int b = 0; b < kStageBlocks; ++b) {
            uint32_t regs[16];
            expand_block<CODEC, decltype(large)::value>(payload + stage + b * Cfg::kBlockQ, first[b], second[b], regs);
            if (b == 0 && !slot_is_free()) return;
            tmem_st16(slot_cols + b * 16, regs);
          }
        };
        if (small_scales<CODEC>(first, second)) expand(std::false_type());
        else expand(std::true_type());
        if (!ok) break;
      }
      __syncwarp();
      if (lane == hands_back) mbar_arrive(&w_empty[w.at]);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[slot.at]);
      w.skip(kDequantGroups);
      slot.skip(kDequantGroups);
      if (behind >= 0) freed.skip(kDequantGroups);
      else if (behind + kDequantGroups > 0) freed.skip(behind + kDequantGroups);
      behind += kDequantGroups;
    }
    const int r = (a.tile0 + tile) * kRows + row;
    if constexpr (Cfg::kExact) {
      // ---------------------------------------------------------------- the last stage's products, then both groups' sums
      static_assert(AS == kDequantGroups, "a group owns a slot");
      if (ok && behind >= 0 && wait_warp(&done[freed.at], freed.parity, abort_flag)) {
        tc_fence_after();
        const int valid = min(kStageBlocks, a.kblocks - (s0 + behind) * kStageBlocks);
#pragma unroll
        for (int b = 0; b < kStageBlocks; ++b) {
          if (b >= valid) break;
          uint32_t products[USED];
          load_products(my_products + (uint32_t)(b * NV), products);
          tmem_wait_ld();
          add_block(products, scale[b]);
        }
      }
      chain_wait();  // outputs, residual and scratch may still be in use by the kernel before this one
      float* mine = reinterpret_cast<float*>(smem) + row;
      dequant_barrier();  // both groups have read their last stage: the rings are free
      if (group == 1)
#pragma unroll
        for (int v = 0; v < USED; ++v) mine[v * kRows] = sums[v];
      dequant_barrier();
      if (group == 0)
#pragma unroll
        for (int v = 0; v < USED; ++v) {
          const float sum = sums[v] + mine[v * kRows];
          if (a.deferred) a.scratch[((size_t)split * NV + v) * a.rows_padded + r] = sum;
          else mine[v * kRows] = sum;
        }
    } else if (chain_wait(); wait_warp(d_full, 0, abort_flag)) {
      // ---------------------------------------------------------------- accumulator out of TMEM (half of it per group)
      // (outputs, residual and scratch may be in use by the kernel before this one until its end)
      tc_fence_after();
      // to the consumer's partial sums, or to this CTA's shared memory (the rings are free: every stage has been read)
      float* dst = a.deferred ? a.scratch + (size_t)split * NV * a.rows_padded + r : reinterpret_cast<float*>(smem) + row;
      const size_t stride = a.deferred ? a.rows_padded : kRows;
#pragma unroll 1
      for (int v0 = group * 16; v0 < NV && v0 < a.vectors; v0 += 16 * kDequantGroups) {
        uint32_t acc[16];
        tmem_ld16(tmem + lane_base + (uint32_t)v0, acc);
        tmem_wait_ld();
#pragma unroll
        for (int v = 0; v < 16; ++v) dst[(size_t)(v0 + v) * stride] = __uint_as_float(acc[v]);
      }
    }
  } else if (warp == kWeightWarp) {
    // ------------------------------------------------------------------ weight loader (one lane)
    if (elect_one()) {
      Ring<WS> w;
      int issued = 0;
      for (int i = 0; i < n; ++i) {
        if (!mbar_wait(&w_empty[w.at], w.parity ^ 1u, abort_flag)) break;
        const int kb = (s0 + i) * kStageBlocks;
        const uint32_t valid = (uint32_t)min(kStageBlocks, a.kblocks - kb);
        const size_t block = (size_t)tile * a.kblocks + kb;
        unsigned char* dst = w_ring + (size_t)w.at * Cfg::kStageW;
        mbar_arrive_expect_tx(&w_full[w.at], valid * (Cfg::kBlockQ + Cfg::kBlockS));
        bulk_copy_g2s(dst, a.quants + block * Cfg::kBlockQ, valid * Cfg::kBlockQ, &w_full[w.at]);
        bulk_copy_g2s(dst + Cfg::kStageQ, a.scales + block * Cfg::kBlockS, valid * Cfg::kBlockS, &w_full[w.at]);
        issued = i + 1;
        w.next();
      }
      if (*abort_flag)  // give up: this warp's own copies land (bounded) before shared memory is released
        for (int i = max(0, issued - WS); i < issued; ++i)
          for (unsigned spin = 0; spin < (1u << 20) && !mbar_try_wait(&w_full[i % WS], (uint32_t)(i / WS) & 1u); ++spin) __nanosleep(64);
    }
  } else if (warp == kActivationWarp) {
    // ------------------------------------------------------------------ activation loader
    if (Cfg::kExact && !a.xh) {
      // Up to kDirectVectors f32 vectors, converted on the way (a launch less): the warp fetches cells of eight columns for as
      // many stages as four cells per lane cover, then fills their buffers one by one. The rows of absent vectors keep stale
      // bytes, which reach no other vector's products.
      chain_wait();  // the activations come from the kernel before this one
      Ring<BS> b;
      Ring<DONE> freed;  // the stage BS before this one
      constexpr int CELLS = 4 * kStageBlocks;  // of a vector in a stage
      const int per_stage = CELLS * a.vectors, stages = 2 * kDirectVectors / a.vectors, K = a.kblocks * 32;
      bool ok = true;
      for (int i0 = 0; i0 < n && ok; i0 += stages) {
        float4 lo[4], hi[4];
        int stage[4], cell[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int e = lane + 32 * j, kg = e % CELLS, v = e % per_stage / CELLS;
          const int column = (s0 + i0 + e / per_stage) * kStageBlocks * 32 + kg * 8;
          stage[j] = e / per_stage < stages && column < K ? e / per_stage : -1;
          cell[j] = (kg * NV + v) * 16;
          if (stage[j] >= 0) {
            const float4* src = reinterpret_cast<const float4*>(a.x + (size_t)v * K + column);
            lo[j] = src[0];
            hi[j] = src[1];
          }
        }
        for (int t = 0; t < stages && i0 + t < n; ++t) {
          if (i0 + t >= BS) {
            ok = wait_warp(&done[freed.at], freed.parity, abort_flag);
            if (!ok) break;
            freed.next();
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (stage[j] == t) {
              const uint2 l = pack4(lo[j]), h = pack4(hi[j]);
              *reinterpret_cast<uint4*>(b_ring + (size_t)b.at * Cfg::kStageB + cell[j]) = make_uint4(l.x, l.y, h.x, h.y);
            }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads through the async proxy
          __syncwarp();
          if (lane == 0) mbar_arrive(&b_full[b.at]);
          b.next();
        }
      }
    } else if (elect_one()) {
      chain_wait();  // the activations come from the kernel before this one
      Ring<BS> b;
      Ring<DONE> freed;  // the stage BS before this one
      int issued = 0;
      for (int i = 0; i < n; ++i) {
        if (i >= BS) {
          if (!mbar_wait(&done[freed.at], freed.parity, abort_flag)) break;
          freed.next();
        }
        const int kb = (s0 + i) * kStageBlocks, groups = min(kStageBlocks, a.kblocks - kb) * 4;  // of eight columns
        unsigned char* dst = b_ring + (size_t)b.at * Cfg::kStageB;
        if (Cfg::kExact && a.xh_nv != NV) {  // the first rows of a wider layout
          mbar_arrive_expect_tx(&b_full[b.at], (uint32_t)groups * NV * 16u);
          for (int kg = 0; kg < groups; ++kg) bulk_copy_g2s(dst + kg * NV * 16, a.xh + ((size_t)kb * 4 + kg) * a.xh_nv * 8, NV * 16u, &b_full[b.at]);
        } else {
          mbar_arrive_expect_tx(&b_full[b.at], (uint32_t)groups * NV * 16u);
          bulk_copy_g2s(dst, a.xh + (size_t)kb * 4 * NV * 8, (uint32_t)groups * NV * 16u, &b_full[b.at]);
        }
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
      Ring<DONE> report;
      bool ok = true;
      const uint64_t desc0 = make_b_desc(smem_u32(b_ring), NV * 16u, 128u);
      for (int i = 0; i < n && ok; ++i) {
        ok = mbar_wait(&b_full[b.at], b.parity, abort_flag) && mbar_wait(&a_full[slot.at], slot.parity, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const int valid = min(kStageBlocks, a.kblocks - (s0 + i) * kStageBlocks);
        // two K = 16 instructions per block: two column groups of B, 8 TMEM columns of A each. Whole stages are unrolled:
        // with constant steps the operands stay in uniform registers (58 cycles per instruction in a loop, 16 unrolled)
        const uint64_t desc = desc0 + (uint64_t)(b.at * (int)(Cfg::kStageB / 16));
        const uint32_t a_cols = a_tmem + (uint32_t)(slot.at * kStageBlocks * 16);
        if constexpr (Cfg::kExact) {
          const uint32_t d_cols = tmem + (uint32_t)(slot.at * kStageBlocks * NV);
#pragma unroll
          for (int j = 0; j < 2 * kStageBlocks; ++j)
            if (j < 2 * valid) umma_ts(d_cols + (uint32_t)(j / 2 * NV), a_cols + 8u * j, desc + 2u * NV * j, kIdesc, j & 1);
          tc_commit(&done[report.at]);
          b.next();
          slot.next();
          report.next();
          continue;
        }
        umma_ts(tmem, a_cols, desc, kIdesc, i > 0 ? 1u : 0u);
        if (valid == kStageBlocks) {
#pragma unroll
          for (int j = 1; j < 2 * kStageBlocks; ++j) umma_ts(tmem, a_cols + 8u * j, desc + 2u * NV * j, kIdesc, 1u);
        } else {
          for (int j = 1; j < 2 * valid; ++j) umma_ts(tmem, a_cols + 8u * j, desc + 2u * NV * j, kIdesc, 1u);
        }
        tc_commit(&done[report.at]);
        b.next();
        slot.next();
        report.next();
      }
      if (ok && !Cfg::kExact) tc_commit(d_full);
    }
  }
  __syncwarp();
  tc_fence_before();
  if (!a.deferred) {
    // ------------------------------------------------------------------ the tile's CTAs add up and finish
    cg::cluster_group cluster = cg::this_cluster();
    if (gridDim.x > 1) cluster.sync();
    else __syncthreads();
    if (!*abort_flag) {
      chain_wait();
      const int ranks = gridDim.x, per = (a.vectors + ranks - 1) / ranks;  // this CTA's share of the vectors
      const int v_lo = split * per, v_hi = min(a.vectors, v_lo + per);
      const int row0 = (a.tile0 + tile) * kRows;
      auto sum4 = [&](int v, int quad) {
        const float* mine = reinterpret_cast<const float*>(smem) + v * kRows + 4 * quad;
        float4 sum = *reinterpret_cast<const float4*>(ranks == 1 ? mine : cluster.map_shared_rank(mine, 0));
        for (int p = 1; p < ranks; ++p) sum = add4(sum, *reinterpret_cast<const float4*>(cluster.map_shared_rank(mine, p)));
        if (a.bias) {
          const int r = row0 + 4 * quad;
          sum = add4(sum, make_float4(r < a.rows ? a.bias[r] : 0.f, r + 1 < a.rows ? a.bias[r + 1] : 0.f, r + 2 < a.rows ? a.bias[r + 2] : 0.f,
                                      r + 3 < a.rows ? a.bias[r + 3] : 0.f));
        }
        return sum;
      };
      if (a.epilogue == ETC_EPILOGUE_SWIGLU) {
        // rows are interleaved in groups of 8: quads 0, 1 of every four are gate rows, 2, 3 their up rows
        for (int i = threadIdx.x; i < (v_hi - v_lo) * 16; i += kStreamThreads) {
          const int v = v_lo + (i >> 4), q = (i & 15), gate = (q >> 1) * 4 + (q & 1);
          const float4 g = sum4(v, gate), u = sum4(v, gate + 2);
          const int c = row0 / 2 + 4 * q;
          if (c < a.rows / 2)
            store4(a, v, c, 4, a.rows / 2,
                   make_float4(silu_tanh(g.x) * u.x, silu_tanh(g.y) * u.y, silu_tanh(g.z) * u.z, silu_tanh(g.w) * u.w));
        }
      } else {
        for (int i = threadIdx.x; i < (v_hi - v_lo) * 32; i += kStreamThreads) {
          const int v = v_lo + (i >> 5), q = i & 31, r = row0 + 4 * q, inside = min(4, a.rows - r);
          if (inside <= 0) continue;
          float4 val = sum4(v, q);
          if (a.epilogue == ETC_EPILOGUE_RESIDUAL) {
            const float* res = a.residual + (size_t)v * a.rows + r;
            val = add4(make_float4(res[0], inside > 1 ? res[1] : 0.f, inside > 2 ? res[2] : 0.f, inside > 3 ? res[3] : 0.f), val);
          }
          store4(a, v, r, inside, a.rows, val);
        }
      }
    }
    if (gridDim.x > 1) cluster.sync();  // the other CTAs may still be reading this one's shared memory
  }
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicCAS(a.status, 0ull, 3ull);  // a bounded wait expired
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::kTmemCols);
  }
}

template <int CODEC, int NV, int USED = NV>
cudaError_t launch_stream_pass(const StreamArgs& args, int tiles, int splits, cudaStream_t stream) {
  constexpr size_t smem = StreamCfg<CODEC, NV>::kSmemBytes;
  auto kernel = qlinear_stream_kernel<CODEC, NV, USED>;
  const cudaError_t attr = opt_in_shared_memory(kernel, smem);
  if (attr != cudaSuccess) return attr;
  return launch_chained_cluster(kernel, dim3((unsigned)splits, (unsigned)tiles), dim3(kStreamThreads), smem, stream, args.deferred ? 1u : (unsigned)splits, args);
}

}  // namespace

int stream_max_vectors() { return 128; }

StreamPlan plan_stream(const TiledWeight& w, int64_t vectors, int sm_count, bool deferred) {
  StreamPlan p;
  const int sms = std::max(1, sm_count);
  const bool exact = vectors <= kExactVectors && w.n_segments == 0 && (w.codec == 2 || w.codec == 8);
  p.nv = exact ? kExactVectors : vectors <= 32 ? 32 : (vectors <= 64 ? 64 : 128);
  p.tiles = (int)(w.rows_padded / kRows);
  p.stages = (int)((w.columns / 32 + kStageBlocks - 1) / kStageBlocks);
  p.xh_bytes = ((size_t)(w.columns / 8) * p.nv * 16 + 255) & ~(size_t)255;
  if (deferred) {
    // as many splits as fit at two CTAs per SM (one at 128 vectors), of at least two stages: the consumer's sum costs little
    // per split, and a shape's sums keep their order whoever computes them
    const int splits = std::min(std::max(1, sms * (p.nv <= 64 ? 2 : 1) / p.tiles), std::max(1, p.stages / 2));
    p.stages_per_split = (p.stages + splits - 1) / splits;
  } else {
    // In stages: those of the fullest SM less what its CTAs expand ahead of the activations (one and a half each), a third more
    // for a CTA that has an SM for itself (nothing overlaps its waits), and a cluster's exchange, which grows with the vectors.
    // Clusters are powers of two (three or six CTAs pack a GPC badly) and are used while all of them are resident at once
    // ([128256 x 4096] takes 73 us with one CTA per tile, 96 with two); those of four and more fill seven eighths of the places at
    // most, and a second wave costs more than they give ([9216 x 1024] x 1 to 32 in fours 8.9 to 11.4 us, in pairs 5.3 to 7.3).
    // Every choice was measured back to back over 2 to 224 tiles, 4 to 224 stages, 1 to 100 vectors and four codecs: this rule's
    // is 0.9 % from the best on average (with a floor of half a stage and a wave more instead 1.8, without the work done ahead 5.5).
    const double exchange = p.nv <= 16 ? 0.75 : p.nv == 32 ? 2.0 : p.nv == 64 ? 2.25 : 3.5;
    double best = 1e30;
    for (int s = 1, log = 0; s <= std::min(kMaxStreamCluster, std::max(1, p.stages / 2)) && (s == 1 || p.tiles * s <= 2 * sms); s *= 2, ++log) {
      if (s >= 4 && p.tiles * s > 2 * sms * 7 / 8) break;
      const int per = (p.stages + s - 1) / s, ctas = (p.tiles * s + sms - 1) / sms;
      const double cost = ctas * std::max(per - 1.5, 1.0) * (ctas > 1 ? 1.0 : 1.33) + log * exchange + (s > 1 && ctas > 1 ? 0.5 : 0.0);
      if (cost < best) { best = cost; p.stages_per_split = per; }
    }
  }
  p.splits = (p.stages + p.stages_per_split - 1) / p.stages_per_split;
  p.deferred = deferred && p.splits > 1;
  p.scratch_bytes = p.deferred ? (size_t)p.splits * p.nv * w.rows_padded * sizeof(float) : 0;
  return p;
}

size_t stream_scratch_bytes(const TiledWeight& w, int64_t vectors, int sm_count) {
  const StreamPlan p = plan_stream(w, vectors, sm_count, true);
  return p.xh_bytes + p.scratch_bytes;
}

cudaError_t launch_qlinear_stream(const TiledWeight& w, const float* x, const __half* xh_ready, int64_t vectors, const float* bias,
                                  const float* residual, int epilogue, float* out, __half* out_xh, void* scratch, DeviceStatus* status,
                                  int sm_count, cudaStream_t stream, int* launches, int xh_nv, DeferredSum* defer) {
  if (defer) *defer = DeferredSum();
  const StreamPlan plan = plan_stream(w, vectors, sm_count, defer && !bias && !out_xh && epilogue != ETC_EPILOGUE_SWIGLU);
  const int K = (int)w.columns;
  __half* xh = reinterpret_cast<__half*>(scratch);
  float* partials = reinterpret_cast<float*>(reinterpret_cast<char*>(scratch) + plan.xh_bytes);
  const bool exact = plan.nv == kExactVectors;
  const bool ready = xh_ready != nullptr && (exact || plan.nv == xh_nv);  // the producer stored the f16 layout with this row stride
  cudaError_t e;
  // Converting on the way saves a launch (2 us, and 3 us of host time) and slows the stream by some 8 %: even at about 64
  // stages per SM (18 us of Q4_0).
  const bool direct = !ready && exact && vectors <= kDirectVectors && (int64_t)plan.tiles * plan.stages <= 64 * (int64_t)sm_count;
  if (!ready && !x) return cudaErrorInvalidValue;
  if (!ready && !direct) {
    e = launch_hand_off_convert(x, vectors, K, plan.nv, xh, sm_count, stream);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  StreamArgs args;
  args.xh = ready ? xh_ready : direct ? nullptr : xh;
  args.x = x;
  args.xh_nv = ready ? xh_nv : plan.nv;
  args.bias = bias;
  args.residual = residual;
  args.out = out;
  args.scratch = partials;
  args.status = &status->code;
  args.out_xh = vectors <= xh_nv ? out_xh : nullptr;
  args.out_xh_nv = xh_nv;
  args.vectors = (int)vectors;
  args.rows = (int)w.rows;
  args.rows_padded = (int)w.rows_padded;
  args.kblocks = K / 32;
  args.epilogue = epilogue;
  args.stages = plan.stages;
  args.stages_per_split = plan.stages_per_split;
  args.deferred = plan.deferred;
  // one launch per run of equal codecs; all of them share the plan of the whole weight
  for (int sgm = 0; sgm < std::max(1, w.n_segments); ++sgm) {
    int codec = w.codec, tiles = plan.tiles;
    args.quants = w.quants;
    args.scales = reinterpret_cast<const unsigned char*>(w.scales);
    args.tile0 = 0;
    if (w.n_segments > 0) {
      const TiledSegment& seg = w.segments[sgm];
      codec = seg.codec;
      tiles = seg.tiles;
      args.tile0 = seg.tile0;
      args.quants += seg.quant_offset;
      args.scales += seg.scale_offset;
    }
    auto pass = [&](auto nv_tag) {
      constexpr int NV = decltype(nv_tag)::value;
      if constexpr (NV == kExactVectors)
        if (args.vectors <= 8) return codec == 2 ? launch_stream_pass<2, NV, 8>(args, tiles, plan.splits, stream) : launch_stream_pass<8, NV, 8>(args, tiles, plan.splits, stream);
      if (codec == 2) return launch_stream_pass<2, NV>(args, tiles, plan.splits, stream);
      if (codec == 8) return launch_stream_pass<8, NV>(args, tiles, plan.splits, stream);
      if constexpr (NV != kExactVectors) {
        if (codec == 12) return launch_stream_pass<12, NV>(args, tiles, plan.splits, stream);
        if (codec == 13) return launch_stream_pass<13, NV>(args, tiles, plan.splits, stream);
        return launch_stream_pass<14, NV>(args, tiles, plan.splits, stream);  // 14, and 11 whose re-cut form is the same
      }
      return cudaErrorInvalidValue;
    };
    e = exact ? pass(std::integral_constant<int, kExactVectors>()) : plan.nv == 32 ? pass(std::integral_constant<int, 32>()) : plan.nv == 64 ? pass(std::integral_constant<int, 64>()) : pass(std::integral_constant<int, 128>());
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  if (plan.deferred) {
    // the consumer sums the partials itself (and adds the residual stream where the epilogue asks for it)
    defer->partials = partials;
    defer->splits = plan.splits;
    defer->vpad = plan.nv;
    defer->rows_padded = (int)w.rows_padded;
  }
  return cudaSuccess;
}

}  // namespace etc
