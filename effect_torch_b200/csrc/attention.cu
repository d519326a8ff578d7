// Paged KV kernels for sm_100a: page-pool append (all four tiers), reference-order attention in
// f64, tensor-core flash-decoding over the block table with split-KV merge, RoPE and append inside
// both for a decoder's one-token steps, and as a kernel of their own for chunks.
//
// Replaces kv_attention_into of the reference (crates/runtime-cpu/src/napi/mod.rs:3320-3565):
// the scatter (:3397-3459) and the attend loop (:3461-3542), and the slab tiers of
// crates/runtime-cpu/src/pool.rs:20-257.
//
// HBM layout (chosen for the B200, not the reference's token-major slab): per layer one K and
// one V slab of [pages][kv_heads][block_size][head_dim] elements, so the block_size rows of one
// (page, head) are one contiguous run (4 KiB for f16, 16 tokens, D=128) that a warp fetches
// with 16-byte cp.async copies. u8 tier scales are [pages][kv_heads][block_size] f32.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "activation.cuh"
#include "chain.cuh"
#include "kernels.h"

namespace etc {

enum : int { kKvF32 = 0, kKvF16 = 1, kKvBF16 = 2, kKvU8 = 3 };

__device__ __forceinline__ size_t pool_elem(const PoolView& p, int page, int head, int slot) {
  return (((size_t)page * p.kv_heads + head) * p.block_size + slot) * p.head_dim;
}
__device__ __forceinline__ size_t pool_scale_index(const PoolView& p, int page, int head, int slot) {
  return ((size_t)page * p.kv_heads + head) * p.block_size + slot;
}

// Widening read of one cached element (pool.rs:51-58; the u8 tier applies (code-128)*scale as
// napi/mod.rs:3474-3476 does).
__device__ __forceinline__ float pool_load(const PoolView& p, const void* slab, const float* scales, size_t elem,
                                           size_t scale_index) {
  switch (p.dtype) {
    case kKvF32: return reinterpret_cast<const float*>(slab)[elem];
    case kKvF16: return __half2float(reinterpret_cast<const __half*>(slab)[elem]);
    case kKvBF16: return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(slab)[elem]);
    default: return __fmul_rn(__fsub_rn((float)reinterpret_cast<const uint8_t*>(slab)[elem], 128.0f), scales[scale_index]);
  }
}

// --------------------------------------------------------------------------------------------
// KV append: grid (tokens, kv_heads, batch), one CTA per (lane, head, new token) row.
// k/v are f32 with explicit strides so both the reference layout [B,Hkv,T,D] and the fused
// projection output [B, ...] can be scattered. u8 tier: scale = absmax/127 + 1e-12,
// code = clamp(round(x/scale), +-127) + 128 with round = ties away from zero (pool.rs:224-240).
// --------------------------------------------------------------------------------------------
__global__ void kv_append_kernel(PoolView pool, const float* __restrict__ k, const float* __restrict__ v,
                                 const LaneInfo* __restrict__ lanes, const int* __restrict__ tables, int64_t lane_stride,
                                 int64_t head_stride, int64_t token_stride) {
  __shared__ float red[2][32];
  const int token = blockIdx.x, head = blockIdx.y, lane_id = blockIdx.z;
  const LaneInfo info = lanes[lane_id];
  if (token >= info.advance) return;  // padded lane or dead row of the chunk
  const int pos = info.cursor + token;
  const int page = tables[info.table_offset + pos / pool.block_size];
  const int slot = pos % pool.block_size;
  const size_t dst = pool_elem(pool, page, head, slot);
  const float* ksrc = k + lane_id * lane_stride + head * head_stride + token * token_stride;
  const float* vsrc = v + lane_id * lane_stride + head * head_stride + token * token_stride;
  const int D = pool.head_dim;
  if (pool.dtype == kKvU8) {
    float kmax = 0.0f, vmax = 0.0f;
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
      kmax = fmaxf(kmax, fabsf(ksrc[d]));
      vmax = fmaxf(vmax, fabsf(vsrc[d]));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      kmax = fmaxf(kmax, __shfl_xor_sync(0xffffffffu, kmax, off));
      vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
    }
    if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = kmax; red[1][threadIdx.x >> 5] = vmax; }
    __syncthreads();
    kmax = 0.0f; vmax = 0.0f;
    for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) { kmax = fmaxf(kmax, red[0][w]); vmax = fmaxf(vmax, red[1][w]); }
    const float kscale = __fadd_rn(__fdiv_rn(kmax, 127.0f), 1e-12f);
    const float vscale = __fadd_rn(__fdiv_rn(vmax, 127.0f), 1e-12f);
    if (threadIdx.x == 0) {
      const size_t si = pool_scale_index(pool, page, head, slot);
      pool.k_scale[si] = kscale;
      pool.v_scale[si] = vscale;
    }
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
      float kc = roundf(__fdiv_rn(ksrc[d], kscale));
      float vc = roundf(__fdiv_rn(vsrc[d], vscale));
      kc = fminf(fmaxf(kc, -127.0f), 127.0f) + 128.0f;
      vc = fminf(fmaxf(vc, -127.0f), 127.0f) + 128.0f;
      reinterpret_cast<uint8_t*>(pool.k)[dst + d] = (uint8_t)kc;
      reinterpret_cast<uint8_t*>(pool.v)[dst + d] = (uint8_t)vc;
    }
    return;
  }
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const float kv = ksrc[d], vv = vsrc[d];
    if (pool.dtype == kKvF32) {
      reinterpret_cast<float*>(pool.k)[dst + d] = kv;
      reinterpret_cast<float*>(pool.v)[dst + d] = vv;
    } else if (pool.dtype == kKvF16) {
      reinterpret_cast<__half*>(pool.k)[dst + d] = __float2half_rn(kv);
      reinterpret_cast<__half*>(pool.v)[dst + d] = __float2half_rn(vv);
    } else {
      reinterpret_cast<__nv_bfloat16*>(pool.k)[dst + d] = __float2bfloat16_rn(kv);
      reinterpret_cast<__nv_bfloat16*>(pool.v)[dst + d] = __float2bfloat16_rn(vv);
    }
  }
}

cudaError_t launch_kv_append(const PoolView& pool, const float* k, const float* v, const LaneInfo* lanes,
                             const int* tables, int batch, int tokens, int64_t lane_stride, int64_t head_stride,
                             int64_t token_stride, cudaStream_t stream) {
  if (batch == 0 || tokens == 0) return cudaSuccess;
  dim3 grid((unsigned)tokens, (unsigned)pool.kv_heads, (unsigned)batch);
  const int threads = std::min(128, ((pool.head_dim + 31) / 32) * 32);
  kv_append_kernel<<<grid, threads, 0, stream>>>(pool, k, v, lanes, tables, lane_stride, head_stride, token_stride);
  return cudaGetLastError();
}

// --------------------------------------------------------------------------------------------
// Reference-order attention. One CTA per (query head, query row, lane). Scores are f64 dot
// products accumulated over the head dimension in index order (the products of two f32 values are
// exact in f64, so this equals the reference's sum bit for bit), scaled, max-reduced; the weights
// exp(s*scale - max) are kept in a global f64 scratch row; then thread c accumulates column c of
// the output over positions in order with separate multiply and add, exactly like the
// reference's loop, and divides by the denominator it accumulated the same way.
// Only exp() can differ from the host libm, by an ulp of f64.
//
// Latency-bound: two dependent f64 chains, head_dim long (scores) and context long (output). What is not part of them is
// kept off them: block-table look-ups and their divisions are done once per position, K rows and V elements are fetched
// four and eight at a time ahead of the adds, weights of contexts up to kExactKept stay in shared memory.
// --------------------------------------------------------------------------------------------
constexpr int kExactKept = 2048;

template <int DTYPE>
__device__ __forceinline__ float exact_load(const void* slab, size_t elem, float scale) {
  if (DTYPE == kKvF32) return reinterpret_cast<const float*>(slab)[elem];
  if (DTYPE == kKvF16) return __half2float(reinterpret_cast<const __half*>(slab)[elem]);
  if (DTYPE == kKvBF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(slab)[elem]);
  return __fmul_rn(__fsub_rn((float)reinterpret_cast<const uint8_t*>(slab)[elem], 128.0f), scale);
}

// `tokens_first`: q and out are [B, tokens, Hq, D] (the fused projection's order) instead of [B, Hq, tokens, D].
template <int DTYPE>
__global__ void __launch_bounds__(128) attention_exact_kernel(PoolView pool, const float* q,
                                                              const LaneInfo* lanes,
                                                              const int* tables, int q_heads, int tokens,
                                                              double scale, long long op_window, float* out,
                                                              double* scratch, int max_ctx, int tokens_first) {
  extern __shared__ float q_s[];  // the query row
  __shared__ double kept[kExactKept];
  __shared__ int row_of[kExactKept];  // (page * kv_heads + head) * block_size + slot of each position
  __shared__ double red[4];
  chain_release();
  chain_wait();
  const int head = blockIdx.x, query = blockIdx.y, lane_id = blockIdx.z;
  const LaneInfo info = lanes[lane_id];
  const int D = pool.head_dim;
  const size_t row_index = ((size_t)lane_id * q_heads + head) * tokens + query;
  const size_t io = (tokens_first ? ((size_t)lane_id * tokens + query) * q_heads + head : row_index) * D;
  float* orow = out + io;
  if (info.advance == 0) {  // padded lane: output stays zero (napi/mod.rs:3371-3372)
    for (int d = threadIdx.x; d < D; d += blockDim.x) orow[d] = 0.0f;
    return;
  }
  const int kv_head = head / (q_heads / pool.kv_heads);
  const int needed = info.cursor + info.advance;
  const int end = min(info.cursor + query + 1, needed);
  int begin = info.start;
  if (op_window >= 0) begin = max((int)max((long long)end - op_window, 0ll), info.start);
  const int span = max(end - begin, 0);
  for (int d = threadIdx.x; d < D; d += blockDim.x) q_s[d] = q[io + d];
  const bool keep = span <= kExactKept;
  double* wrow = keep ? kept : scratch + row_index * (size_t)max_ctx;
  const int* table = tables + info.table_offset;
  auto find_row = [&](int i) {
    const int pos = begin + i, block = pos / pool.block_size;
    return (table[block] * pool.kv_heads + kv_head) * pool.block_size + (pos - block * pool.block_size);
  };
  auto row_at = [&](int i) { return keep ? row_of[i] : find_row(i); };
  auto k_scale = [&](int row) { return DTYPE == kKvU8 ? pool.k_scale[row] : 0.0f; };
  auto v_scale = [&](int row) { return DTYPE == kKvU8 ? pool.v_scale[row] : 0.0f; };
  __syncthreads();

  double local_max = -INFINITY;
  for (int i = threadIdx.x; i < span; i += blockDim.x) {
    const int row = find_row(i);
    if (keep) row_of[i] = row;
    const size_t base = (size_t)row * D;
    const float ks = k_scale(row);
    double score = 0.0;
    int c = 0;
    for (; c + 4 <= D; c += 4) {
      float kv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) kv[u] = exact_load<DTYPE>(pool.k, base + c + u, ks);
#pragma unroll
      for (int u = 0; u < 4; ++u) score += (double)q_s[c + u] * (double)kv[u];
    }
    for (; c < D; ++c) score += (double)q_s[c] * (double)exact_load<DTYPE>(pool.k, base + c, ks);
    const double scaled = __dmul_rn(score, scale);
    wrow[i] = scaled;
    local_max = fmax(local_max, scaled);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) local_max = fmax(local_max, __shfl_xor_sync(0xffffffffu, local_max, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local_max;
  __syncthreads();
  const double maximum = fmax(fmax(red[0], red[1]), fmax(red[2], red[3]));
  for (int i = threadIdx.x; i < span; i += blockDim.x) wrow[i] = exp(__dsub_rn(wrow[i], maximum));
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    double result = 0.0, denominator = 0.0;
    int i = 0;
    for (; i + 8 <= span; i += 8) {
      float value[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int row = row_at(i + u);
        value[u] = exact_load<DTYPE>(pool.v, (size_t)row * D + c, v_scale(row));
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const double w = wrow[i + u];
        result = __dadd_rn(result, __dmul_rn(w, (double)value[u]));
        denominator = __dadd_rn(denominator, w);
      }
    }
    for (; i < span; ++i) {
      const int row = row_at(i);
      const double w = wrow[i];
      result = __dadd_rn(result, __dmul_rn(w, (double)exact_load<DTYPE>(pool.v, (size_t)row * D + c, v_scale(row))));
      denominator = __dadd_rn(denominator, w);
    }
    orow[c] = (float)__ddiv_rn(result, denominator);
  }
}

cudaError_t launch_attention_exact(const PoolView& pool, const float* q, const LaneInfo* lanes, const int* tables,
                                   int batch, int q_heads, int tokens, double scale, long long op_window, float* out,
                                   double* scratch, int max_ctx, cudaStream_t stream, bool tokens_first) {
  if (batch == 0 || tokens == 0) return cudaSuccess;
  auto launch = [&](auto kernel) {
    return launch_chained(kernel, dim3((unsigned)q_heads, (unsigned)tokens, (unsigned)batch), dim3(128), (size_t)pool.head_dim * sizeof(float), stream, pool,
                          q, lanes, tables, q_heads, tokens, scale, op_window, out, scratch, max_ctx, (int)tokens_first);
  };
  switch (pool.dtype) {
    case kKvF32: return launch(attention_exact_kernel<kKvF32>);
    case kKvF16: return launch(attention_exact_kernel<kKvF16>);
    case kKvBF16: return launch(attention_exact_kernel<kKvBF16>);
    default: return launch(attention_exact_kernel<kKvU8>);
  }
}

// The same for one-token steps of the decoder with an f32 cache whose contexts fit in shared memory, RoPE and append included. A
// CTA per (query head, lane) fetches the cached rows, which were written before this step, and the angles before it waits for
// the projection; then it rotates its query and the new K row, which all query heads of a KV head do and the first of them
// stores. K rows are padded so that a warp's 16-byte reads of 32 positions do not conflict. Two launches (9.2 us with its
// 4-byte loads of K from memory at one line per thread, 1.8 us for RoPE) in one of 4 at contexts of 32 to 95.
constexpr size_t kExactStepSmem = 200 * 1024;
static int exact_step_slots(int max_ctx) { return (max_ctx + 3) & ~3; }  // keeps what follows them 16-byte aligned
static size_t exact_step_smem(int head_dim, int max_ctx) {
  return (size_t)exact_step_slots(max_ctx) * ((2 * head_dim + 4) * sizeof(float) + sizeof(double)) + 2 * head_dim * sizeof(double);
}

__global__ void __launch_bounds__(128) attention_exact_step_kernel(PoolView pool, const float* qkv, const LaneInfo* lanes, const int* tables,
                                                                   const double* inv_freq, int layout, int q_heads, double scale,
                                                                   long long op_window, float* out, int slots) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[4];
  const int D = pool.head_dim, half = D / 2, pitch = D + 4;
  double* q_s = reinterpret_cast<double*>(smem);                     // [D]
  double2* angle = reinterpret_cast<double2*>(q_s + D);              // [D / 2] (sine, cosine)
  double* weight_s = reinterpret_cast<double*>(angle + half);        // [slots], a multiple of 4
  float* k_s = reinterpret_cast<float*>(weight_s + slots);           // [slots][pitch]
  float* v_s = k_s + (size_t)slots * pitch;                          // [slots][D]
  chain_release();
  const int head = blockIdx.x, lane_id = blockIdx.y, group = q_heads / pool.kv_heads, kv_head = head / group;
  const LaneInfo info = lanes[lane_id];
  float* orow = out + ((size_t)lane_id * q_heads + head) * D;
  if (info.advance == 0) {  // padded lane: output stays zero (napi/mod.rs:3371-3372)
    chain_wait();
    for (int d = threadIdx.x; d < D; d += blockDim.x) orow[d] = 0.0f;
    return;
  }
  const int end = info.cursor + 1;
  const int begin = op_window >= 0 ? max((int)max((long long)end - op_window, 0ll), info.start) : info.start;
  const int cached = min(max(end - begin, 0), slots) - 1;  // positions before the new one
  const int* table = tables + info.table_offset;
  auto row_of = [&](int pos) {
    const int block = pos / pool.block_size;
    return ((size_t)table[block] * pool.kv_heads + kv_head) * pool.block_size + (pos - block * pool.block_size);
  };
  const int quads = D / 4;
  for (int i = threadIdx.x; i < cached * quads; i += blockDim.x) {
    const int at = i / quads, c = 4 * (i - at * quads);
    const size_t src = row_of(begin + at) * D + c;
    const unsigned kd = (unsigned)__cvta_generic_to_shared(k_s + at * pitch + c), vd = (unsigned)__cvta_generic_to_shared(v_s + at * D + c);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(kd), "l"(reinterpret_cast<const float*>(pool.k) + src) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vd), "l"(reinterpret_cast<const float*>(pool.v) + src) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int j = threadIdx.x; j < half; j += blockDim.x) {
    double s, c;
    sincos((double)info.cursor * inv_freq[j], &s, &c);
    angle[j] = make_double2(s, c);
  }
  __syncthreads();  // the angles
  chain_wait();
  const size_t fresh = row_of(info.cursor) * D;
  const bool stores = head == kv_head * group;
  const float* row = qkv + (size_t)lane_id * (q_heads + 2 * pool.kv_heads) * D;
  for (int i = threadIdx.x; i < 3 * half; i += blockDim.x) {
    const int what = i / half, j = i - what * half;  // 0: query, 1: key, 2: value
    const int i0 = layout == 0 ? j : 2 * j, i1 = layout == 0 ? half + j : 2 * j + 1;
    const float* src = row + (size_t)(what == 0 ? head : q_heads + (what - 1) * pool.kv_heads + kv_head) * D;
    float r0 = src[i0], r1 = src[i1];
    if (what < 2) {
      const double first = (double)r0, second = (double)r1, s = angle[j].x, c = angle[j].y;
      r0 = (float)__dsub_rn(__dmul_rn(first, c), __dmul_rn(second, s));
      r1 = (float)__dadd_rn(__dmul_rn(second, c), __dmul_rn(first, s));
    }
    if (what == 0) {
      q_s[i0] = (double)r0;
      q_s[i1] = (double)r1;
      continue;
    }
    float* dst = what == 1 ? k_s + (size_t)cached * pitch : v_s + (size_t)cached * D;
    dst[i0] = r0;
    dst[i1] = r1;
    if (stores) {
      float* slab = reinterpret_cast<float*>(what == 1 ? pool.k : pool.v) + fresh;
      slab[i0] = r0;
      slab[i1] = r1;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int span = cached + 1;
  double local_max = -INFINITY;
  for (int i = threadIdx.x; i < span; i += blockDim.x) {
    const float4* k4 = reinterpret_cast<const float4*>(k_s + (size_t)i * pitch);
    double score = 0.0;
#pragma unroll 4
    for (int c = 0; c < quads; ++c) {
      const float4 k = k4[c];
      score += q_s[4 * c] * (double)k.x;  // exact products: contracted or not, one rounding per term
      score += q_s[4 * c + 1] * (double)k.y;
      score += q_s[4 * c + 2] * (double)k.z;
      score += q_s[4 * c + 3] * (double)k.w;
    }
    const double scaled = __dmul_rn(score, scale);
    weight_s[i] = scaled;
    local_max = fmax(local_max, scaled);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) local_max = fmax(local_max, __shfl_xor_sync(0xffffffffu, local_max, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local_max;
  __syncthreads();
  const double maximum = fmax(fmax(red[0], red[1]), fmax(red[2], red[3]));
  for (int i = threadIdx.x; i < span; i += blockDim.x) weight_s[i] = exp(__dsub_rn(weight_s[i], maximum));
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    double result = 0.0, denominator = 0.0;
#pragma unroll 8
    for (int i = 0; i < span; ++i) {
      const double w = weight_s[i];
      result = __dadd_rn(result, __dmul_rn(w, (double)v_s[(size_t)i * D + c]));
      denominator = __dadd_rn(denominator, w);
    }
    orow[c] = (float)__ddiv_rn(result, denominator);
  }
}

// Many lanes of long contexts leave one or two CTAs to an SM, which wait for their rows wave after wave; from some number of CTAs
// per SM on the two launches, which read the rows where they are, are as fast or faster. Whole steps of four layers, one launch and
// two, by CTAs per SM: 64 columns, one CTA at a time 7 610 and 673 us, 14 969 and 990, 21 1292 and 1243, 28 1602 and 1549 (two
// at a time: 28 1159 and 1456); 32 columns 14 1431 and 1417, 21 1997 and 1871; 128 columns, one at a time 10 1178 and
// 1301, 14 1398 and 1316, 28 2441 and 2180; two at a time 10 815 and 987, 14 1157 and 1013, 28 1497 and 1471.
bool attention_exact_step_supported(const PoolView& pool, int batch, int q_heads, int max_ctx, int sm_count) {
  const size_t smem = exact_step_smem(pool.head_dim, max_ctx);
  if (pool.dtype != kKvF32 || pool.kv_heads <= 0 || q_heads % pool.kv_heads != 0 || pool.head_dim % 4 != 0 || smem > kExactStepSmem) return false;
  const int at_once = (int)(kSmSharedBytes / (smem + kCtaSharedReserve));
  const int64_t ctas = (int64_t)batch * q_heads;
  return pool.head_dim >= 128 ? at_once > 2 || ctas <= 12ll * sm_count : at_once > 1 || ctas <= 16ll * sm_count;
}

cudaError_t launch_attention_exact_step(const PoolView& pool, const float* qkv, const LaneInfo* lanes, const int* tables, const double* inv_freq, int layout,
                                        int batch, int q_heads, double scale, long long op_window, float* out, int max_ctx, cudaStream_t stream) {
  if (batch == 0) return cudaSuccess;
  const cudaError_t attr = opt_in_shared_memory(attention_exact_step_kernel, kExactStepSmem);
  if (attr != cudaSuccess) return attr;
  return launch_chained(attention_exact_step_kernel, dim3((unsigned)q_heads, (unsigned)batch), dim3(128), exact_step_smem(pool.head_dim, max_ctx), stream, pool,
                        qkv, lanes, tables, inv_freq, layout, q_heads, scale, op_window, out, exact_step_slots(max_ctx));
}

// --------------------------------------------------------------------------------------------
// Tensor-core flash-decoding (one query token per lane, f16 or bf16 pages of 16 tokens).
//
// Grid (splits, kv_heads, batch); a CTA of 4 warps serves one (lane, kv head, page range) and all
// G = q_heads/kv_heads query heads of that KV head at once: the G query rows are rows 0..G-1 of
// the m16n8k16 A operand, so every K/V page is fetched from HBM once per KV head, not once per
// query head. Warps take pages round-robin; each warp keeps a 3-deep cp.async ring of
// (K page, V page) in shared memory (16-byte copies, XOR-swizzled so ldmatrix is conflict-free),
// computes S = Q K^T with mma.sync, the online softmax in registers (exp2 domain, scale*log2(e)
// folded into Q), P V with mma.sync reusing the S accumulators as the A operand, and at the end
// the 4 warps merge their (m, l, O) through shared memory. With splits > 1 the CTA writes an
// unnormalised partial (m, l, O) per query head and attention_merge_kernel combines the splits.
//
// FUSED (the decoder's one-token steps): the CTA also does what rope_append_kernel does for its heads. It adds up the fused
// q/k/v projection's split-K partials of its G query heads (every split of a lane does, they are a few KB from L2), rotates
// them, and the CTA whose range holds the new token's page rotates and stores the new K and V rows. Cached rows, lanes and
// tables were written before this step, so all pages but the new token's, and the angles, are on their way before the wait for
// the projection. One launch and its chain of L2 round trips less per layer (RoPE alone took 3.6 us of a 65 us layer).
//
// Roofline: HBM-bound: bytes = sum_lanes ctx * 2 * kv_heads * D * sizeof(kv) (+ q, out, tables).
// --------------------------------------------------------------------------------------------
constexpr int kAttnWarps = 4;
constexpr int kAttnStages = 3;
constexpr int kPageTokens = 16;

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem_src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem_ptr) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(smem_ptr);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem_ptr) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(smem_ptr);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (BF16) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if (BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

struct AttnArgs {
  const void* k;
  const void* v;
  const float* k_scale;    // u8 tier: one f32 per (page, head, slot)
  const float* v_scale;
  const float* q;          // [B, Hq, D] f32
  const LaneInfo* lanes;
  const int* tables;
  float* out;              // [B, Hq, D] f32 (splits == 1)
  __half* out_xh;          // optional f16 copy of out in the hand-off layout: the o-projection's B operand
  int out_xh_nv;
  float* partial;          // [B, Hq, splits, D + 2] f32: O unnormalised, then m (log2 domain), l
  int q_heads, kv_heads;
  int pages_per_split;
  int tokens;              // query tokens per lane (1: decode; > 1: a prefill chunk, q and out are [B, tokens, Hq, D])
  float scale_log2;        // scale * log2(e)
  long long op_window;
};
// fused RoPE and append: the projection's rows [B, q heads | k heads | v heads, D] (or their split-K partials)
struct FusedAttnArgs : AttnArgs {
  const float* qkv;
  DeferredSum sum;
  const double* inv_freq;
  int rope_layout;
  void *slab[2];           // K and V again, to store the new rows
  float *slab_scale[2];
};

// smem per warp per stage: K page then V page, each 16 rows x D*2 bytes, 16-byte chunk c of row r
// stored at chunk (c ^ (r & 7)) within its 128-byte group.
template <int D>
__device__ __forceinline__ int swizzled_offset(int row, int chunk) {  // in bytes
  return row * (D * 2) + ((chunk & ~7) | ((chunk ^ row) & 7)) * 16;
}

// The same for a page of code bytes: rows of D bytes, conflict free for ldmatrix over eight rows.
template <int D>
__device__ __forceinline__ int swizzled_bytes(int row, int chunk) {
  return row * D + (chunk ^ (D == 128 ? row & 7 : (row >> 1) & 3)) * 16;
}

// Four bytes b0..b3 -> halves 1024 + b, minus 1152 = b - 128 (exact).
template <unsigned LO = 0x4140, unsigned HI = 0x4342>  // which two bytes go into lo, and into hi
__device__ __forceinline__ void bytes_to_half2(uint32_t w, uint32_t& lo, uint32_t& hi) {
  const __half2 bias = __floats2half2_rn(1152.0f, 1152.0f);
  uint32_t lo_bits = __byte_perm(w, 0x64646464u, LO), hi_bits = __byte_perm(w, 0x64646464u, HI);
  const __half2 l = __hsub2(*reinterpret_cast<__half2*>(&lo_bits), bias), h = __hsub2(*reinterpret_cast<__half2*>(&hi_bits), bias);
  lo = *reinterpret_cast<const uint32_t*>(&l);
  hi = *reinterpret_cast<const uint32_t*>(&h);
}

// SORTED: the lane with `rank` longer ones before it (of equals, the first first), by a CTA that has a thread per lane. CTAs
// start in the order of their index, so that the longest lanes do not start last and run on alone. 64 lanes of 128 to 4096
// tokens x 8 heads 98.8 -> 90 us (1.00 of the copy bandwidth).
constexpr int kMaxSortedLanes = kAttnWarps * 32;
__device__ __forceinline__ int lane_by_length(const LaneInfo* lanes, int n, int rank) {
  extern __shared__ __align__(128) unsigned char smem[];  // not in use yet
  int* lengths = reinterpret_cast<int*>(smem);
  const int t = threadIdx.x;
  if (t < n) {
    const LaneInfo info = lanes[t];
    lengths[t] = info.advance > 0 ? info.cursor - info.start : -1;
  }
  __syncthreads();
  if (t < n) {
    const int mine = lengths[t];
    int before = 0;
    for (int j = 0; j < n; ++j) before += lengths[j] > mine || (lengths[j] == mine && j < t);
    if (before == rank) lengths[kMaxSortedLanes] = t;
  }
  __syncthreads();
  const int found = lengths[kMaxSortedLanes];
  __syncthreads();  // before the first copies overwrite it
  return __shfl_sync(0xffffffffu, found, 0);
}

// U8: the int8 tier (code - 128) * scale with one scale per cached row (napi/mod.rs:3474-3476): pages travel as bytes, and the
// row scales multiply the score columns (K) and the probabilities before P V (V), so the tensor core only ever sees exact small
// integers. ldmatrix hands a thread four code bytes at a time, which it widens to two f16 pairs in registers: of K the columns
// 4 t .. 4 t + 3 of a row, which become the operand's columns 2 t, 2 t + 1, 2 t + 8 and 2 t + 9 (the query fragments are
// permuted alike, inside each sum of 16); of V, transposed, two columns of two rows, which go to two neighbouring output tiles
// (columns 2 n and 2 n + 1 of every 16).
template <int D, bool BF16, bool U8, bool FUSED, bool SORTED>
__global__ void __launch_bounds__(kAttnWarps * 32) attention_mma_kernel(std::conditional_t<FUSED, FusedAttnArgs, AttnArgs> a) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int RAW_PAGE = kPageTokens * D * (U8 ? 1 : 2);      // one page as cached
  constexpr int SCALE_BYTES = U8 ? kPageTokens * 4 : 0;         // its row scales
  constexpr int STAGE_BYTES = 2 * (RAW_PAGE + SCALE_BYTES);
  constexpr int WARP_BYTES = kAttnStages * STAGE_BYTES;         // a warp's ring
  constexpr int CHUNKS = D / 8;    // 16-byte chunks per row
  constexpr int KSTEPS = D / 16;   // k16 steps of the QK^T product
  constexpr int DTILES = D / 8;    // n-tiles of the PV product
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  if (!FUSED) chain_wait();
  const int split = blockIdx.x, kv_head = blockIdx.y;
  const int lane_id = SORTED ? lane_by_length(a.lanes, gridDim.z, blockIdx.z) : blockIdx.z;
  const LaneInfo info = a.lanes[lane_id];
  const int G = a.q_heads / a.kv_heads;
  const int nsplits = gridDim.x;
  const int end = info.cursor + info.advance;
  int begin = info.start;
  if (a.op_window >= 0) begin = max((int)max((long long)end - a.op_window, 0ll), info.start);
  const bool idle_lane = info.advance == 0 || end <= begin;
  // page range of this split (pages are indexed from the table start, i.e. position 0)
  const int first_page = begin / kPageTokens;
  const int last_page = idle_lane ? first_page : (end - 1) / kPageTokens + 1;  // exclusive
  const int p0 = first_page + split * a.pages_per_split;
  const int p1 = min(last_page, p0 + a.pages_per_split);
  const int new_page = last_page - 1;  // FUSED: of the token that this step appends, the last page of the warp that has it

  unsigned char* my_smem = smem + (size_t)warp * WARP_BYTES;
  const int* table = a.tables + info.table_offset;
  const size_t page_stride = (size_t)a.kv_heads * RAW_PAGE;  // bytes between consecutive pages
  const unsigned char* kbase = reinterpret_cast<const unsigned char*>(a.k) + (size_t)kv_head * RAW_PAGE;
  const unsigned char* vbase = reinterpret_cast<const unsigned char*>(a.v) + (size_t)kv_head * RAW_PAGE;

  // SORTED: the warp's page numbers, 32 at a time, one per lane: the copies then wait for a shuffle instead of a table look-up
  // each (of an address that is not known to be uniform: 30 % of a page's time).
  int held_from = p0 + warp;
  auto look_up = [&] {
    const int at = held_from + lane * kAttnWarps;
    return at < p1 ? table[at] : 0;
  };
  int held = SORTED ? look_up() : 0;
  auto page_of = [&](int page_index) {
    if (!SORTED) return table[page_index];
    if (page_index >= held_from + 32 * kAttnWarps) {
      held_from += 32 * kAttnWarps;
      held = look_up();
    }
    return __shfl_sync(0xffffffffu, held, (page_index - held_from) / kAttnWarps);
  };

  auto issue = [&](int page_index, int stage, bool but_new = false) {
    if (page_index < p1 && !(FUSED && but_new && page_index == new_page)) {
      const int page = page_of(page_index);
      const size_t off = (size_t)page * page_stride;
      unsigned char* ks = my_smem + stage * STAGE_BYTES;
      unsigned char* vs = ks + RAW_PAGE;
      if (U8) {
        // the bytes, then the 16 row scales of K and of V
#pragma unroll
        for (int i = 0; i < RAW_PAGE / 16 / 32; ++i) {
          const int c = lane + 32 * i, so = swizzled_bytes<D>(c / (D / 16), c % (D / 16));
          cp_async16(ks + so, kbase + off + (size_t)c * 16);
          cp_async16(vs + so, vbase + off + (size_t)c * 16);
        }
        if (lane < 8) {
          const size_t si = ((size_t)page * a.kv_heads + kv_head) * kPageTokens;  // 16 floats = 4 chunks each
          const float* src = (lane < 4 ? a.k_scale : a.v_scale) + si + (lane & 3) * 4;
          cp_async16(my_smem + stage * STAGE_BYTES + 2 * RAW_PAGE + lane * 16, src);
        }
      } else {
#pragma unroll
        for (int i = 0; i < (kPageTokens * CHUNKS) / 32; ++i) {
          const int c = lane + 32 * i;  // chunk index within the page
          const int row = c / CHUNKS, chunk = c % CHUNKS;
          const int so = swizzled_offset<D>(row, chunk);
          cp_async16(ks + so, kbase + off + (size_t)c * 16);
          cp_async16(vs + so, vbase + off + (size_t)c * 16);
        }
      }
    }
    cp_async_commit();  // always commit so group counting stays uniform
  };
  // this warp's pages: p0 + warp, p0 + warp + 4, ...; the first copies are in flight while the query rows are fetched
  int next_issue = p0 + warp;
#pragma unroll
  for (int s = 0; s < kAttnStages - 1; ++s) {
    issue(next_issue, s, true);
    next_issue += kAttnWarps;
  }

  // fused: query rows 0..G-1 of this KV head, [G][D] f32, in a ring stage that the loop fills last
  // (U8: behind the rings)
  float* q_rows = reinterpret_cast<float*>(smem + (U8 ? kAttnWarps * WARP_BYTES : (kAttnStages - 1) * STAGE_BYTES));
  if constexpr (FUSED) {
    constexpr int HALF = D / 2, STEP = kAttnWarps * 32 / HALF, ITEMS = 3, IN_FLIGHT = 8;
    __shared__ double2 angle[HALF];  // (sine, cosine) per pair
    __shared__ float fresh[2][D];    // the new K row, the new V row
    const int j = threadIdx.x % HALF, h0 = threadIdx.x / HALF;
    const bool works = p0 < p1, appends = works && new_page < p1;
    if (works && h0 == 0) {
      double sine, cosine;
      sincos((double)info.cursor * a.inv_freq[j], &sine, &cosine);
      angle[j] = make_double2(sine, cosine);
    }
    chain_wait();
    if (works) {  // the same for the whole CTA
      const int i0 = a.rope_layout == 0 ? j : 2 * j, i1 = a.rope_layout == 0 ? HALF + j : 2 * j + 1;
      const int heads = a.q_heads + 2 * a.kv_heads, mine = appends ? G + 2 : G;
      auto head_of = [&](int h) { return h < G ? kv_head * G + h : a.q_heads + (h - G) * a.kv_heads + kv_head; };
      const size_t split_stride = (size_t)a.sum.vpad * a.sum.rows_padded;
      const int splits = max(a.sum.splits, 1);  // one "split": the finished rows
      const float* rows = a.sum.splits > 0 ? a.sum.partials + (size_t)lane_id * a.sum.rows_padded : a.qkv + (size_t)lane_id * heads * D;
      __syncthreads();  // the angles
      const double sine = angle[j].x, cosine = angle[j].y;
      for (int hb = h0; hb < mine; hb += STEP * ITEMS) {
        float x0[ITEMS], x1[ITEMS];
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) x0[u] = x1[u] = 0.0f;
        for (int s0 = 0; s0 < splits; s0 += IN_FLIGHT) {
          float part0[ITEMS][IN_FLIGHT], part1[ITEMS][IN_FLIGHT];
#pragma unroll
          for (int u = 0; u < ITEMS; ++u)
#pragma unroll
            for (int t = 0; t < IN_FLIGHT; ++t)
              if (hb + u * STEP < mine && s0 + t < splits) {
                const float* src = rows + (size_t)(s0 + t) * split_stride + (size_t)head_of(hb + u * STEP) * D;
                part0[u][t] = src[i0];
                part1[u][t] = src[i1];
              }
#pragma unroll
          for (int u = 0; u < ITEMS; ++u)
#pragma unroll
            for (int t = 0; t < IN_FLIGHT; ++t)
              if (hb + u * STEP < mine && s0 + t < splits) {
                x0[u] += part0[u][t];
                x1[u] += part1[u][t];
              }
        }
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
          const int h = hb + u * STEP;
          if (h >= mine) break;
          float r0 = x0[u], r1 = x1[u];
          if (h <= G) {  // not the value row
            const double first = (double)r0, second = (double)r1;
            r0 = (float)__dsub_rn(__dmul_rn(first, cosine), __dmul_rn(second, sine));
            r1 = (float)__dadd_rn(__dmul_rn(second, cosine), __dmul_rn(first, sine));
          }
          float* dst = h < G ? q_rows + h * D : fresh[h - G];
          dst[i0] = r0;
          dst[i1] = r1;
        }
      }
      __syncthreads();  // the rows
      if (appends && warp < 2) {  // warp 0 stores K, warp 1 V
        const int slot = info.cursor % kPageTokens;
        const size_t row = ((size_t)table[new_page] * a.kv_heads + kv_head) * kPageTokens + slot;
        void* slab = warp == 0 ? a.slab[0] : a.slab[1];
        const float* src = fresh[warp];
        if (U8) {  // one scale per cached row, as kv_append_kernel (pool.rs:224-240)
          float amax = 0.0f;
#pragma unroll
          for (int d = lane; d < D; d += 32) amax = fmaxf(amax, fabsf(src[d]));
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
          const float scale = __fadd_rn(__fdiv_rn(amax, 127.0f), 1e-12f);
          if (lane == 0) (warp == 0 ? a.slab_scale[0] : a.slab_scale[1])[row] = scale;
#pragma unroll
          for (int d = lane; d < D; d += 32)
            reinterpret_cast<uint8_t*>(slab)[row * D + d] = (uint8_t)(fminf(fmaxf(roundf(__fdiv_rn(src[d], scale)), -127.0f), 127.0f) + 128.0f);
        } else {
#pragma unroll
          for (int d = 2 * lane; d < D; d += 64) reinterpret_cast<uint32_t*>(slab)[(row * D + d) / 2] = pack2<BF16>(src[d], src[d + 1]);
        }
      }
    }
  }

  // Q fragments: rows 0..G-1 = query heads of this KV head, scaled into the exp2 domain
  uint32_t qf[KSTEPS][4];
  {
    const bool lo_ok = g < G, hi_ok = g + 8 < G;
    const float* qrow_lo = FUSED ? q_rows + (lo_ok ? g : 0) * D : a.q + ((size_t)lane_id * a.q_heads + kv_head * G + (lo_ok ? g : 0)) * D;
    const float* qrow_hi = FUSED ? q_rows + (hi_ok ? g + 8 : 0) * D : a.q + ((size_t)lane_id * a.q_heads + kv_head * G + (hi_ok ? g + 8 : 0)) * D;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
      const int c0 = ks * 16 + (U8 ? 4 : 2) * t, c1 = c0 + (U8 ? 2 : 8);
      float2 x0 = lo_ok ? *reinterpret_cast<const float2*>(qrow_lo + c0) : make_float2(0.f, 0.f);
      float2 x1 = hi_ok ? *reinterpret_cast<const float2*>(qrow_hi + c0) : make_float2(0.f, 0.f);
      float2 x2 = lo_ok ? *reinterpret_cast<const float2*>(qrow_lo + c1) : make_float2(0.f, 0.f);
      float2 x3 = hi_ok ? *reinterpret_cast<const float2*>(qrow_hi + c1) : make_float2(0.f, 0.f);
      qf[ks][0] = pack2<BF16>(x0.x * a.scale_log2, x0.y * a.scale_log2);
      qf[ks][1] = pack2<BF16>(x1.x * a.scale_log2, x1.y * a.scale_log2);
      qf[ks][2] = pack2<BF16>(x2.x * a.scale_log2, x2.y * a.scale_log2);
      qf[ks][3] = pack2<BF16>(x3.x * a.scale_log2, x3.y * a.scale_log2);
    }
  }
  if constexpr (FUSED) {
    __syncthreads();  // the query rows have been read, the new rows are stored
    // the new token's page where it is among the first ones of its warp
#pragma unroll
    for (int s = 0; s < kAttnStages - 1; ++s)
      if (p0 + warp + s * kAttnWarps == new_page) issue(new_page, s);
  }

  float o[DTILES][4];
#pragma unroll
  for (int i = 0; i < DTILES; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[i][j] = 0.0f;
  float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.0f, l_hi = 0.0f;  // rows g and g+8

  int stage = 0;
  for (int page_index = p0 + warp; page_index < p1; page_index += kAttnWarps) {
    issue(next_issue, (stage + kAttnStages - 1) % kAttnStages);
    next_issue += kAttnWarps;
    if (FUSED && page_index == new_page) cp_async_wait<0>();  // it may have been requested out of turn
    else cp_async_wait<kAttnStages - 1>();
    __syncwarp();
    const unsigned char* ks_page = my_smem + stage * STAGE_BYTES;
    const unsigned char* vs_page = ks_page + RAW_PAGE;
    const float* page_scales = reinterpret_cast<const float*>(my_smem + stage * STAGE_BYTES + 2 * RAW_PAGE);  // U8: K rows, then V rows

    // S = Q K^T : two n-tiles of 8 tokens
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
    if constexpr (U8) {
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ks += 2) {
        uint32_t codes[4], b0, b1;  // step ks: rows 0-7, rows 8-15; step ks + 1
        ldmatrix_x4(codes, ks_page + swizzled_bytes<D>((lane & 7) + (((lane >> 3) & 1) << 3), ks + (lane >> 4)));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          bytes_to_half2(codes[2 * u], b0, b1);
          mma_16816<BF16>(s0, qf[ks + u], b0, b1);
          bytes_to_half2(codes[2 * u + 1], b0, b1);
          mma_16816<BF16>(s1, qf[ks + u], b0, b1);
        }
      }
    } else {
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ++ks) {
        uint32_t kf[4];
        const int row = (lane & 7) + ((lane >> 4) << 3);
        const int chunk = 2 * ks + ((lane >> 3) & 1);
        ldmatrix_x4(kf, ks_page + swizzled_offset<D>(row, chunk));
        mma_16816<BF16>(s0, qf[ks], kf[0], kf[1]);
        mma_16816<BF16>(s1, qf[ks], kf[2], kf[3]);
      }
    }
    if (U8) {  // score of token column c carries that cached row's K scale
      const float ka0 = page_scales[2 * t], ka1 = page_scales[2 * t + 1], kb0 = page_scales[2 * t + 8], kb1 = page_scales[2 * t + 9];
      s0[0] *= ka0; s0[1] *= ka1; s0[2] *= ka0; s0[3] *= ka1;
      s1[0] *= kb0; s1[1] *= kb1; s1[2] *= kb0; s1[3] *= kb1;
    }
    // mask positions outside [begin, end)
    const int base_pos = page_index * kPageTokens;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int pa = base_pos + 2 * t + j, pb = pa + 8;
      if (pa < begin || pa >= end) s0[j] = s0[2 + j] = -INFINITY;
      if (pb < begin || pb >= end) s1[j] = s1[2 + j] = -INFINITY;
    }
    // online softmax for rows g (index 0,1) and g+8 (index 2,3)
    float mx_lo = fmaxf(fmaxf(s0[0], s0[1]), fmaxf(s1[0], s1[1]));
    float mx_hi = fmaxf(fmaxf(s0[2], s0[3]), fmaxf(s1[2], s1[3]));
    mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1));
    mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
    mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1));
    mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
    const float mn_lo = fmaxf(m_lo, mx_lo), mn_hi = fmaxf(m_hi, mx_hi);
    // a page with every position masked leaves the running maximum at -inf: keep factors finite
    const float alpha_lo = mn_lo == -INFINITY ? 1.0f : exp2f(m_lo - mn_lo);
    const float alpha_hi = mn_hi == -INFINITY ? 1.0f : exp2f(m_hi - mn_hi);
    const float sub_lo = mn_lo == -INFINITY ? 0.0f : mn_lo, sub_hi = mn_hi == -INFINITY ? 0.0f : mn_hi;
    float p0v[4], p1v[4];
    p0v[0] = exp2f(s0[0] - sub_lo); p0v[1] = exp2f(s0[1] - sub_lo);
    p0v[2] = exp2f(s0[2] - sub_hi); p0v[3] = exp2f(s0[3] - sub_hi);
    p1v[0] = exp2f(s1[0] - sub_lo); p1v[1] = exp2f(s1[1] - sub_lo);
    p1v[2] = exp2f(s1[2] - sub_hi); p1v[3] = exp2f(s1[3] - sub_hi);
    l_lo = l_lo * alpha_lo + (p0v[0] + p0v[1] + p1v[0] + p1v[1]);
    l_hi = l_hi * alpha_hi + (p0v[2] + p0v[3] + p1v[2] + p1v[3]);
    m_lo = mn_lo; m_hi = mn_hi;
    if (U8) {  // V row scales ride on the probabilities; the denominators above stay unscaled
      const float* vsc = page_scales + kPageTokens;
      const float va0 = vsc[2 * t], va1 = vsc[2 * t + 1], vb0 = vsc[2 * t + 8], vb1 = vsc[2 * t + 9];
      p0v[0] *= va0; p0v[1] *= va1; p0v[2] *= va0; p0v[3] *= va1;
      p1v[0] *= vb0; p1v[1] *= vb1; p1v[2] *= vb0; p1v[3] *= vb1;
    }
    uint32_t pf[4];
    pf[0] = pack2<BF16>(p0v[0], p0v[1]);  // row g,   tokens 2t, 2t+1
    pf[1] = pack2<BF16>(p0v[2], p0v[3]);  // row g+8
    pf[2] = pack2<BF16>(p1v[0], p1v[1]);  // row g,   tokens 2t+8, 2t+9
    pf[3] = pack2<BF16>(p1v[2], p1v[3]);
    // O = O * alpha + P V
    auto accumulate = [&](float (&acc)[4], uint32_t b0, uint32_t b1) {
      acc[0] *= alpha_lo; acc[1] *= alpha_lo; acc[2] *= alpha_hi; acc[3] *= alpha_hi;
      mma_16816<BF16>(acc, pf, b0, b1);
    };
#pragma unroll
    for (int dp = 0; dp < DTILES / 2; dp += U8 ? 2 : 1) {
      uint32_t vf[4];
      const int row = (lane & 7) + (((lane >> 3) & 1) << 3);
      if constexpr (U8) {  // columns 16 dp .. 16 dp + 31: rows 0-7 and 8-15 of the first 16, then of the others
        ldmatrix_x4_trans(vf, vs_page + swizzled_bytes<D>(row, dp + (lane >> 4)));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint32_t even0, odd0, even1, odd1;
          bytes_to_half2<0x4240, 0x4341>(vf[2 * u], even0, odd0);
          bytes_to_half2<0x4240, 0x4341>(vf[2 * u + 1], even1, odd1);
          accumulate(o[2 * (dp + u)], even0, even1);
          accumulate(o[2 * (dp + u) + 1], odd0, odd1);
        }
      } else {
        const int chunk = 2 * dp + (lane >> 4);
        ldmatrix_x4_trans(vf, vs_page + swizzled_offset<D>(row, chunk));
        accumulate(o[2 * dp], vf[0], vf[1]);
        accumulate(o[2 * dp + 1], vf[2], vf[3]);
      }
    }
    __syncwarp();
    stage = (stage + 1) % kAttnStages;
  }
  cp_async_wait<0>();
  // quad-reduce the denominators (each lane summed its own token columns)
  l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1);
  l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
  l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1);
  l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);

  // ---- merge the 4 warps through shared memory (reusing the page ring)
  __syncthreads();
  float* mo = reinterpret_cast<float*>(smem);          // [warp][16 rows][D]
  float* mm = mo + kAttnWarps * 16 * D;                // [warp][16]
  float* ml = mm + kAttnWarps * 16;                    // [warp][16]
#pragma unroll
  for (int i = 0; i < DTILES; ++i) {
    // U8: tiles 2 n and 2 n + 1 hold the even and the odd columns of 16
    const int c0 = U8 ? i / 2 * 16 + 4 * t + (i & 1) : i * 8 + 2 * t, c1 = c0 + (U8 ? 2 : 1);
    float* lo = mo + ((size_t)warp * 16 + g) * D;
    float* hi = lo + 8 * D;
    lo[c0] = o[i][0]; lo[c1] = o[i][1];
    hi[c0] = o[i][2]; hi[c1] = o[i][3];
  }
  if (t == 0) {
    mm[warp * 16 + g] = m_lo; mm[warp * 16 + g + 8] = m_hi;
    ml[warp * 16 + g] = l_lo; ml[warp * 16 + g + 8] = l_hi;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += blockDim.x) {
    const int row = idx / D, d = idx - row * D;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) m = fmaxf(m, mm[w * 16 + row]);
    float acc = 0.0f, l = 0.0f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float mw = mm[w * 16 + row];
      const float f = mw == -INFINITY ? 0.0f : exp2f(mw - m);
      acc += f * mo[((size_t)w * 16 + row) * D + d];
      l += f * ml[w * 16 + row];
    }
    const int head = kv_head * G + row;
    if (nsplits == 1) {
      const float val = l > 0.0f ? acc / l : 0.0f;
      if (a.out) a.out[((size_t)lane_id * a.q_heads + head) * D + d] = val;
      if (a.out_xh) {
        const int k = head * D + d;
        a.out_xh[hand_off_cell(k >> 3, lane_id, a.out_xh_nv, a.q_heads * (D / 8)) + (k & 7)] = half_sat(val);
      }
    } else {
      float* dst = a.partial + (((size_t)lane_id * a.q_heads + head) * nsplits + split) * (D + 2);
      dst[d] = acc;
      if (d == 0) { dst[D] = m; dst[D + 1] = l; }
    }
  }
}

// Combines split partials: out = sum_s 2^(m_s - m) O_s / sum_s 2^(m_s - m) l_s. grid (Hq, B).
__global__ void attention_merge_kernel(const float* partial, int q_heads, int splits, int D,
                                       float* out, __half* out_xh, int xh_nv) {
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  const int head = blockIdx.x, lane_id = blockIdx.y;
  const float* base = partial + ((size_t)lane_id * q_heads + head) * splits * (D + 2);
  // Latency-bound: the outputs of up to 32 splits are requested first, then every split's (m, l), fetched once per CTA;
  // the outputs are added in split order. (With eight in flight, after the factors: 6.3 us for 25 splits of 32 heads, now
  // 4.9.)
  constexpr int IN_FLIGHT = 32;
  extern __shared__ float factor[];  // [splits] 2^(m_s - m), then [splits] l_s
  float p[IN_FLIGHT];
  auto fetch = [&](int s0, int d) {
#pragma unroll
    for (int u = 0; u < IN_FLIGHT; ++u)
      if (s0 + u < splits && d < D) p[u] = base[(size_t)(s0 + u) * (D + 2) + d];
  };
  fetch(0, threadIdx.x);
  float m = -INFINITY;
  for (int s = threadIdx.x & 31; s < splits; s += 32) m = fmaxf(m, base[(size_t)s * (D + 2) + D]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  for (int s = threadIdx.x; s < splits; s += blockDim.x) {
    const float ms = base[(size_t)s * (D + 2) + D];
    factor[s] = ms == -INFINITY ? 0.0f : exp2f(ms - m);
    factor[splits + s] = base[(size_t)s * (D + 2) + D + 1];
  }
  __syncthreads();
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float acc = 0.0f, l = 0.0f;
    for (int s0 = 0; s0 < splits; s0 += IN_FLIGHT) {
      if (s0 > 0 || d != (int)threadIdx.x) fetch(s0, d);
#pragma unroll
      for (int u = 0; u < IN_FLIGHT; ++u) {
        if (s0 + u >= splits) break;
        acc += factor[s0 + u] * p[u];
        l += factor[s0 + u] * factor[splits + s0 + u];
      }
    }
    const float val = l > 0.0f ? acc / l : 0.0f;
    if (out) out[((size_t)lane_id * q_heads + head) * D + d] = val;
    if (out_xh) {
      const int k = head * D + d;
      out_xh[hand_off_cell(k >> 3, lane_id, xh_nv, q_heads * (D / 8)) + (k & 7)] = half_sat(val);
    }
  }
}

// --------------------------------------------------------------------------------------------
// Chunked prefill: T query tokens per lane on top of the cached ones (napi/mod.rs:3420-3477 semantics: token t of the chunk
// attends positions up to cursor + t). Grid (token tiles, kv_heads, batch), longest tiles first. A CTA of 4 warps serves 64
// MMA rows = (token, query head) pairs of 64 / G tokens, 16 rows per warp; the warps walk the lane's pages together, four
// pages (64 positions) at a time, which arrive by cp.async one step ahead in a ring of two stages. Per step a warp does
// S = Q K^T (16 x 64), the online softmax in registers and O += P V with mma.sync.
//
// Bound by the legacy tensor path (a step is 512 mma.sync per CTA at head dim 128, three CTAs per SM). One 16-row tile per
// CTA whose warps took alternate pages and merged at the end read every page four times as often and computed a score in
// twice the instructions.
// --------------------------------------------------------------------------------------------
constexpr int kChunkRows = 64;       // MMA rows per CTA
constexpr int kChunkTokens = 64;     // cached positions per step
constexpr int kChunkPages = kChunkTokens / kPageTokens;

template <int D, bool U8>
struct ChunkCfg {
  static constexpr int kSide = kChunkTokens * D * 2;                 // K or V of a step as MMA operands
  static constexpr int kRawSide = U8 ? kChunkTokens * D : kSide;     // as cached
  static constexpr int kScales = U8 ? 2 * kChunkTokens * 4 : 0;      // row scales of K, then of V
  static constexpr int kStage = 2 * kRawSide + kScales;
  static constexpr size_t kSmemBytes = 2 * (size_t)kStage + (U8 ? 2 * kSide : 0);
};

__device__ __forceinline__ void cp_async16_or_zero(void* smem_dst, const void* gmem_src, bool live) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem_src), "r"(live ? 16 : 0));
}

template <int D, bool BF16, bool U8>
__global__ void __launch_bounds__(128, U8 ? 2 : 3) attention_chunk_kernel(AttnArgs a) {
  using Cfg = ChunkCfg<D, U8>;
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int CHUNKS = D / 8, KSTEPS = D / 16, DTILES = D / 8, NT = kChunkTokens / 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  const int kv_head = blockIdx.y, lane_id = blockIdx.z, T = a.tokens;
  const LaneInfo info = a.lanes[lane_id];
  const int G = a.q_heads / a.kv_heads, tile_tokens = kChunkRows / G;
  const int token0 = (int)(gridDim.x - 1 - blockIdx.x) * tile_tokens, tokens_here = min(tile_tokens, T - token0);
  const int row_lo = warp * 16 + g, row_hi = row_lo + 8;  // this thread's rows; row r is query token r / G, head r % G
  const bool live_lo = row_lo < tokens_here * G, live_hi = row_hi < tokens_here * G;
  const int token_lo = token0 + row_lo / G, token_hi = token0 + row_hi / G;
  auto begin_of = [&](int end) { return a.op_window >= 0 ? max((int)max((long long)end - a.op_window, 0ll), info.start) : info.start; };
  const bool idle = info.advance == 0;
  const int end_lo = live_lo && !idle ? info.cursor + token_lo + 1 : 0, end_hi = live_hi && !idle ? info.cursor + token_hi + 1 : 0;
  const int begin_lo = begin_of(end_lo), begin_hi = begin_of(end_hi);
  // the tile as a whole, and the positions that every row of this warp attends
  const int end = idle ? 0 : info.cursor + token0 + tokens_here, begin = begin_of(idle ? 0 : info.cursor + token0 + 1);
  const int full_begin = begin_of(info.cursor + token0 + min(warp * 16 + 15, tokens_here * G - 1) / G + 1);
  const int full_end = warp * 16 + 15 < tokens_here * G && !idle ? info.cursor + token0 + warp * 16 / G + 1 : 0;
  const int first_page = begin / kPageTokens, last_page = end > begin ? (end - 1) / kPageTokens + 1 : first_page;
  const int steps = (last_page - first_page + kChunkPages - 1) / kChunkPages;

  const int* table = a.tables + info.table_offset;
  constexpr int RAW_PAGE = Cfg::kRawSide / kChunkPages;
  const size_t page_stride = (size_t)a.kv_heads * RAW_PAGE;
  const unsigned char* kbase = reinterpret_cast<const unsigned char*>(a.k) + (size_t)kv_head * RAW_PAGE;
  const unsigned char* vbase = reinterpret_cast<const unsigned char*>(a.v) + (size_t)kv_head * RAW_PAGE;
  auto load = [&](int step) {
    unsigned char* ks = smem + (step & 1) * Cfg::kStage;
    unsigned char* vs = ks + Cfg::kRawSide;
    const int page0 = first_page + step * kChunkPages;
    size_t page[kChunkPages];
#pragma unroll
    for (int p = 0; p < kChunkPages; ++p) page[p] = (size_t)table[min(page0 + p, last_page - 1)];
    constexpr int PER_PAGE = RAW_PAGE / 16;  // 16-byte chunks; pages beyond the last are zeros (0 x NaN is not 0)
#pragma unroll
    for (int p = 0; p < kChunkPages; ++p) {
      const bool live = page0 + p < last_page;
#pragma unroll
      for (int c = threadIdx.x; c < PER_PAGE; c += 128) {
        const size_t src = page[p] * page_stride + (size_t)c * 16;
        const int at = U8 ? (p * PER_PAGE + c) * 16 : swizzled_offset<D>(p * kPageTokens + c / CHUNKS, c % CHUNKS);
        cp_async16_or_zero(ks + at, kbase + src, live);
        cp_async16_or_zero(vs + at, vbase + src, live);
      }
    }
    if (U8 && threadIdx.x < 8 * kChunkPages) {  // 16 f32 scales per page and side: 4 chunks each
      const int p = threadIdx.x >> 3, c = threadIdx.x & 7;
      const size_t si = ((size_t)table[min(page0 + p, last_page - 1)] * a.kv_heads + kv_head) * kPageTokens + (c & 3) * 4;
      cp_async16_or_zero(ks + 2 * Cfg::kRawSide + (c >> 2) * kChunkTokens * 4 + p * kPageTokens * 4 + (c & 3) * 16, (c < 4 ? a.k_scale : a.v_scale) + si,
                         page0 + p < last_page);
    }
    cp_async_commit();
  };
  if (steps > 0) load(0);

  uint32_t qf[KSTEPS][4];
  {
    const float* q_lo = a.q + (((size_t)lane_id * T + (live_lo ? token_lo : 0)) * a.q_heads + kv_head * G + (live_lo ? row_lo % G : 0)) * D;
    const float* q_hi = a.q + (((size_t)lane_id * T + (live_hi ? token_hi : 0)) * a.q_heads + kv_head * G + (live_hi ? row_hi % G : 0)) * D;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
      const int c0 = ks * 16 + 2 * t;
      const float2 x0 = *reinterpret_cast<const float2*>(q_lo + c0), x1 = *reinterpret_cast<const float2*>(q_hi + c0);
      const float2 x2 = *reinterpret_cast<const float2*>(q_lo + c0 + 8), x3 = *reinterpret_cast<const float2*>(q_hi + c0 + 8);
      qf[ks][0] = pack2<BF16>(x0.x * a.scale_log2, x0.y * a.scale_log2);
      qf[ks][1] = pack2<BF16>(x1.x * a.scale_log2, x1.y * a.scale_log2);
      qf[ks][2] = pack2<BF16>(x2.x * a.scale_log2, x2.y * a.scale_log2);
      qf[ks][3] = pack2<BF16>(x3.x * a.scale_log2, x3.y * a.scale_log2);
    }
  }
  float o[DTILES][4];
#pragma unroll
  for (int i = 0; i < DTILES; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[i][j] = 0.0f;
  float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.0f, l_hi = 0.0f;

  for (int step = 0; step < steps; ++step) {
    cp_async_wait<0>();
    __syncthreads();  // this step's pages are in, and every warp is done with the stage that the next load overwrites
    if (step + 1 < steps) load(step + 1);
    const unsigned char* raw = smem + (step & 1) * Cfg::kStage;
    const unsigned char* ks_page = raw;
    const unsigned char* vs_page = raw + Cfg::kRawSide;
    const float* scales = reinterpret_cast<const float*>(raw + 2 * Cfg::kRawSide);
    if (U8) {  // bytes -> f16 integers (code - 128) in the swizzled operand layout; the row scales come in below
      unsigned char* wide = smem + 2 * Cfg::kStage;
      for (int c = threadIdx.x; c < 2 * Cfg::kRawSide / 16; c += 128) {
        const int side = c / (Cfg::kRawSide / 16), cc = c % (Cfg::kRawSide / 16), row = cc / (D / 16), chunk = 2 * (cc % (D / 16));
        const uint4 codes = *reinterpret_cast<const uint4*>(raw + (size_t)c * 16);
        const uint32_t w[4] = {codes.x, codes.y, codes.z, codes.w};
        uint32_t h[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) bytes_to_half2(w[j], h[2 * j], h[2 * j + 1]);
        unsigned char* dst = wide + side * Cfg::kSide;
        *reinterpret_cast<uint4*>(dst + swizzled_offset<D>(row, chunk)) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(dst + swizzled_offset<D>(row, chunk + 1)) = make_uint4(h[4], h[5], h[6], h[7]);
      }
      __syncthreads();
      ks_page = wide;
      vs_page = wide + Cfg::kSide;
    }
    // S = Q K^T: eight n-tiles of 8 positions
    float s[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks)
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        uint32_t kf[4];
        ldmatrix_x4(kf, ks_page + swizzled_offset<D>(n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * ks + ((lane >> 3) & 1)));
        mma_16816<BF16>(s[n], qf[ks], kf[0], kf[1]);
        mma_16816<BF16>(s[n + 1], qf[ks], kf[2], kf[3]);
      }
    const int base = (first_page + step * kChunkPages) * kPageTokens;
    if (U8) {
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const float2 sc = *reinterpret_cast<const float2*>(scales + n * 8 + 2 * t);
        s[n][0] *= sc.x; s[n][1] *= sc.y; s[n][2] *= sc.x; s[n][3] *= sc.y;
      }
    }
    if (base < full_begin || base + kChunkTokens > full_end) {
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int pos = base + n * 8 + 2 * t + j;
          if (pos < begin_lo || pos >= end_lo) s[n][j] = -INFINITY;
          if (pos < begin_hi || pos >= end_hi) s[n][2 + j] = -INFINITY;
        }
    }
    float mx_lo = m_lo, mx_hi = m_hi;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      mx_lo = fmaxf(mx_lo, fmaxf(s[n][0], s[n][1]));
      mx_hi = fmaxf(mx_hi, fmaxf(s[n][2], s[n][3]));
    }
    mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1));
    mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
    mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1));
    mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
    // a row with every position masked so far keeps its maximum at -inf: keep factors finite
    const float sub_lo = mx_lo == -INFINITY ? 0.0f : mx_lo, sub_hi = mx_hi == -INFINITY ? 0.0f : mx_hi;
    const float alpha_lo = exp2f(m_lo - sub_lo), alpha_hi = exp2f(m_hi - sub_hi);
    m_lo = mx_lo; m_hi = mx_hi;
    l_lo *= alpha_lo; l_hi *= alpha_hi;
#pragma unroll
    for (int i = 0; i < DTILES; ++i) { o[i][0] *= alpha_lo; o[i][1] *= alpha_lo; o[i][2] *= alpha_hi; o[i][3] *= alpha_hi; }
    // O += P V, 16 positions at a time
#pragma unroll
    for (int n = 0; n < NT; n += 2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float (&p)[4] = s[n + h];
        p[0] = exp2f(p[0] - sub_lo); p[1] = exp2f(p[1] - sub_lo); p[2] = exp2f(p[2] - sub_hi); p[3] = exp2f(p[3] - sub_hi);
        l_lo += p[0] + p[1];
        l_hi += p[2] + p[3];
        if (U8) {  // V row scales ride on the probabilities; the denominators stay unscaled
          const float2 sc = *reinterpret_cast<const float2*>(scales + kChunkTokens + (n + h) * 8 + 2 * t);
          p[0] *= sc.x; p[1] *= sc.y; p[2] *= sc.x; p[3] *= sc.y;
        }
      }
      const uint32_t pf[4] = {pack2<BF16>(s[n][0], s[n][1]), pack2<BF16>(s[n][2], s[n][3]), pack2<BF16>(s[n + 1][0], s[n + 1][1]),
                              pack2<BF16>(s[n + 1][2], s[n + 1][3])};
#pragma unroll
      for (int dp = 0; dp < DTILES / 2; ++dp) {
        uint32_t vf[4];
        ldmatrix_x4_trans(vf, vs_page + swizzled_offset<D>(n * 8 + (lane & 7) + (((lane >> 3) & 1) << 3), 2 * dp + (lane >> 4)));
        mma_16816<BF16>(o[2 * dp], pf, vf[0], vf[1]);
        mma_16816<BF16>(o[2 * dp + 1], pf, vf[2], vf[3]);
      }
    }
  }
  // quad-reduce the denominators (each lane summed its own columns)
  l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1);
  l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
  l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1);
  l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!(h ? live_hi : live_lo)) continue;
    const float l = h ? l_hi : l_lo, inv = l > 0.0f ? 1.0f / l : 0.0f;
    const size_t row = (size_t)lane_id * T + (h ? token_hi : token_lo);
    const int head = kv_head * G + (h ? row_hi : row_lo) % G;
#pragma unroll
    for (int i = 0; i < DTILES; ++i) {
      const float x = o[i][2 * h] * inv, y = o[i][2 * h + 1] * inv;
      if (a.out) *reinterpret_cast<float2*>(a.out + (row * a.q_heads + head) * D + i * 8 + 2 * t) = make_float2(x, y);
      if (a.out_xh) {
        const __half2 v = half2_sat(x, y);
        *reinterpret_cast<__half2*>(a.out_xh + hand_off_cell(head * (D / 8) + i, row, a.out_xh_nv, a.q_heads * (D / 8)) + 2 * t) = v;
      }
    }
  }
}

template <int D, bool BF16, bool U8>
static cudaError_t launch_attention_chunk_t(const AttnArgs& args, int batch, cudaStream_t stream) {
  constexpr size_t smem = ChunkCfg<D, U8>::kSmemBytes;
  auto kernel = attention_chunk_kernel<D, BF16, U8>;
  const cudaError_t attr = opt_in_shared_memory(kernel, smem);
  if (attr != cudaSuccess) return attr;
  const int tile_tokens = kChunkRows / (args.q_heads / args.kv_heads);
  return launch_chained(kernel, dim3((unsigned)((args.tokens + tile_tokens - 1) / tile_tokens), (unsigned)args.kv_heads, (unsigned)batch), dim3(128), smem, stream,
                        args);
}

bool attention_mma_supported(const PoolView& pool, int q_heads, int tokens) {
  const int G = pool.kv_heads > 0 ? q_heads / pool.kv_heads : 0;
  return tokens >= 1 && pool.block_size == kPageTokens && (pool.head_dim == 64 || pool.head_dim == 128) &&
         (pool.dtype == kKvF16 || pool.dtype == kKvBF16 || pool.dtype == kKvU8) && G >= 1 && G <= 16 && q_heads % pool.kv_heads == 0;
}

AttnPlan plan_attention(int batch, int q_heads, int kv_heads, int head_dim, int max_pages, int sm_count) {
  AttnPlan p;
  const int ctas = std::max(1, batch * kv_heads);
  const int target = std::max(1, sm_count) * 2;
  int splits = std::max(1, target / ctas);
  // Two CTAs per SM and no more. Twice as many from three splits on was slower in all of 4 to 8 sequences (8 KV heads of 128,
  // 512 to 4096 tokens each: f16 4 sequences 12.7 us against 17.1, 8 sequences 21.4 against 26.0, int8 31.9 against 32.7; all
  // of 2048 tokens: 12.5 against 17.2, 17.3 against 21.5, 20.7 against 23.9). Beyond, lengths decide, which this plan does
  // not see: 10 and 13 sequences of mixed lengths gain (int8 35.9 against 25.2, 56.0 against 34.8; f16 22.9 against 22.6, 32.9
  // against 27.8), those of one length lose (24.8 against 28.4, 33.4 against 35.3; 19.8 against 24.2, 23.4 against 28.5).
  // at least 2 pages per warp per split
  splits = std::min(splits, std::max(1, max_pages / (kAttnWarps * 2)));
  p.pages_per_split = std::max(1, (max_pages + splits - 1) / splits);
  p.splits = std::max(1, (max_pages + p.pages_per_split - 1) / p.pages_per_split);
  p.scratch_bytes = p.splits > 1 ? (size_t)batch * q_heads * p.splits * (head_dim + 2) * sizeof(float) : 0;
  p.sm_count = std::max(1, sm_count);
  return p;
}

size_t plan_attention_max_scratch(int batch, int q_heads, int kv_heads, int head_dim, int max_pages, int sm_count) {
  size_t need = 0;
  for (int pages = 1; pages <= max_pages; ++pages)
    need = std::max(need, plan_attention(batch, q_heads, kv_heads, head_dim, pages, sm_count).scratch_bytes);
  return need;
}

template <int D, bool BF16, bool U8, bool FUSED, bool SORTED>
static cudaError_t launch_attention_mma_t(const PoolView& pool, const std::conditional_t<FUSED, FusedAttnArgs, AttnArgs>& args, int batch, int grid_x,
                                          cudaStream_t stream) {
  constexpr size_t page = (size_t)kPageTokens * D * 2;
  constexpr size_t ring = U8 ? (size_t)kAttnWarps * kAttnStages * 2 * (kPageTokens * D + kPageTokens * 4) + (FUSED ? 16 * D * sizeof(float) : 0)
                             : (size_t)kAttnWarps * kAttnStages * 2 * page;
  constexpr size_t merge = (size_t)kAttnWarps * 16 * (D + 2) * sizeof(float);
  constexpr size_t smem = ring > merge ? ring : merge;
  auto kernel = attention_mma_kernel<D, BF16, U8, FUSED, SORTED>;
  const cudaError_t attr = opt_in_shared_memory(kernel, smem);
  if (attr != cudaSuccess) return attr;
  dim3 grid((unsigned)grid_x, (unsigned)pool.kv_heads, (unsigned)batch);
  return launch_chained(kernel, grid, dim3(kAttnWarps * 32), smem, stream, args);
}

cudaError_t launch_attention_mma(const PoolView& pool, const float* q, const LaneInfo* lanes, const int* tables,
                                 int batch, int q_heads, double scale, long long op_window, float* out,
                                 const AttnPlan& plan, float* scratch, cudaStream_t stream, int* launches, __half* out_xh, int xh_nv,
                                 int tokens, const FusedRope* rope) {
  if (batch == 0) return cudaSuccess;
  if (rope && tokens != 1) return cudaErrorInvalidValue;
  FusedAttnArgs args;
  if (rope) {
    args.qkv = rope->qkv;
    args.sum = rope->sum;
    args.inv_freq = rope->inv_freq;
    args.rope_layout = rope->layout;
    args.slab[0] = pool.k;
    args.slab[1] = pool.v;
    args.slab_scale[0] = pool.k_scale;
    args.slab_scale[1] = pool.v_scale;
  }
  args.out_xh = out_xh;
  args.out_xh_nv = xh_nv;
  args.k = pool.k; args.v = pool.v; args.q = q; args.lanes = lanes; args.tables = tables; args.out = out;
  args.partial = scratch; args.q_heads = q_heads; args.kv_heads = pool.kv_heads;
  args.pages_per_split = plan.pages_per_split;
  args.scale_log2 = (float)(scale * 1.4426950408889634);
  args.op_window = op_window;
  args.tokens = tokens;
  args.k_scale = pool.k_scale;
  args.v_scale = pool.v_scale;
  cudaError_t e;
  // the tier and the head width pick the instantiation
  auto launch = [&](auto wide, auto bf16, auto u8) {
    constexpr int D = decltype(wide)::value ? 128 : 64;
    constexpr bool BF16 = decltype(bf16)::value, U8 = decltype(u8)::value;
    if (tokens > 1) return launch_attention_chunk_t<D, BF16, U8>(args, batch, stream);
    // Longest lanes first from half as many CTAs again as an SM holds at once (by shared memory and registers: two of f16 pages of
    // 128 columns, three of bytes, four of 64 columns), where a CTA has up to 32 pages and more for each such round: finding its
    // lane costs every CTA some two microseconds. Without and with it, lanes of equal length and of 3 to 100 % of the longest (8 heads
    // of 128 columns, f16): 64 lanes (1.7 rounds) of 500 tokens 29.7 and 32.2 us, 18.8 and 19.0, of 1000 47.8 and 50.0, 32.5
    // and 31.4, of 4096 159 and 162, 96 and 86; 128 lanes (3.5) of 500 54.7 and 61.3, 34.3 and 42.9, of 2000 161 and
    // 168, 97.6 and 101, with one lane in ten long 61.6 and 53.0, of 4096 312 and 320, 187 and 181, 98.5 and 75.6.
    constexpr int kAtOnce = D == 64 ? 4 : U8 ? 3 : 2;
    const int64_t ctas = (int64_t)batch * pool.kv_heads * plan.splits, places = (int64_t)kAtOnce * plan.sm_count;
    const bool sorted = batch <= kMaxSortedLanes && 2 * ctas >= 3 * places && plan.pages_per_split * places >= 32 * ctas;
    auto decode = [&](auto fused, auto longest_first) {
      return launch_attention_mma_t<D, BF16, U8, decltype(fused)::value, decltype(longest_first)::value>(pool, args, batch, plan.splits, stream);
    };
    if (rope) return sorted ? decode(std::true_type(), std::true_type()) : decode(std::true_type(), std::false_type());
    return sorted ? decode(std::false_type(), std::true_type()) : decode(std::false_type(), std::false_type());
  };
  auto dispatch = [&](auto wide) {
    if (pool.dtype == kKvU8) return launch(wide, std::false_type(), std::true_type());
    if (pool.dtype == kKvBF16) return launch(wide, std::true_type(), std::false_type());
    return launch(wide, std::false_type(), std::false_type());
  };
  e = pool.head_dim == 128 ? dispatch(std::true_type()) : dispatch(std::false_type());
  if (e != cudaSuccess) return e;
  if (launches) ++*launches;
  if (tokens > 1) return cudaSuccess;
  if (plan.splits > 1) {
    dim3 grid((unsigned)q_heads, (unsigned)batch);
    e = launch_chained(attention_merge_kernel, grid, dim3((unsigned)std::min(128, pool.head_dim)), 2 * (size_t)plan.splits * sizeof(float), stream, (const float*)scratch, q_heads, plan.splits,
                       pool.head_dim, out, out_xh, xh_nv);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  return cudaSuccess;
}

// --------------------------------------------------------------------------------------------
// Fused RoPE + KV append. grid (groups of heads, batch, tokens), D/2 threads: token t of lane b is row b*tokens + t
// of qkv, sits at position cursor + t, and its rotated query goes to q_out[b, t, head, :].
// qkv row layout: [q heads | k heads | v heads] x D. Query heads are rotated into q_out, key heads
// are rotated and stored into the pool, value heads are stored. Angles in f64 like rope_kernel.
// --------------------------------------------------------------------------------------------
__device__ __forceinline__ void pool_store(const PoolView& p, void* slab, size_t elem, float value) {
  if (p.dtype == kKvF32) reinterpret_cast<float*>(slab)[elem] = value;
  else if (p.dtype == kKvF16) reinterpret_cast<__half*>(slab)[elem] = __float2half_rn(value);
  else reinterpret_cast<__nv_bfloat16*>(slab)[elem] = __float2bfloat16_rn(value);
}

// A CTA is GROUPS groups of half threads (the pairs of a head), each of which serves HEADS heads. One head per CTA for decode
// steps, whose few rows need every SM and whose chain is short; sixteen for chunks, where the f64 sine and cosine, the same for
// all heads of a row, otherwise dominate (2048 rows x 48 heads: 104 us with one head per CTA).
template <int HEADS, int GROUPS>
__global__ void rope_append_kernel(PoolView pool, const float* qkv, const LaneInfo* lanes,
                                   const int* tables, const double* __restrict__ inv_freq, int layout,
                                   int q_heads, float* q_out, DeferredSum sum) {
  __shared__ double2 angle[GROUPS > 1 ? 64 : 1];  // (sine, cosine) per pair
  __shared__ float red[32];
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  const int lane_id = blockIdx.y, tok = blockIdx.z, tokens = gridDim.z;
  const int D = pool.head_dim, half = D / 2, heads = q_heads + 2 * pool.kv_heads;
  const int width = GROUPS > 1 ? (int)blockDim.x / GROUPS : (int)blockDim.x;  // whole warps
  const int group = GROUPS > 1 ? (int)threadIdx.x / width : 0, pair = (int)threadIdx.x - group * width;
  const bool live = pair < half;  // head dims below 64 leave threads of the warp without a pair
  const int j = live ? pair : 0;
  const size_t row = (size_t)lane_id * tokens + tok;
  const int i0 = layout == 0 ? j : 2 * j, i1 = layout == 0 ? half + j : 2 * j + 1;
  const int head0 = blockIdx.x * HEADS * GROUPS + group;  // this group's heads: head0, head0 + GROUPS, ...
  const double freq = inv_freq[j];
  chain_wait();
  // What the angles and the cells of the cache need, then the heads' inputs, then the angles while those are under way.
  const LaneInfo info = lanes[lane_id];
  const int pos = info.cursor + tok;
  int page = 0, slot = 0;
  if (info.advance > 0 && head0 + (HEADS - 1) * GROUPS >= q_heads) {
    const int block = pos / pool.block_size;
    page = tables[info.table_offset + block];
    slot = pos - block * pool.block_size;
  }
  // The projection may have left its split-K partials unsummed: they are added up here, in split order (a narrow shard of a
  // tensor-parallel group has up to 32 splits; eight loads are in flight at a time).
  constexpr int IN_FLIGHT = 8;
  const bool summing = HEADS * GROUPS == 1 && sum.splits > 0;
  const float* partials = sum.partials + row * sum.rows_padded + (size_t)head0 * D;
  const size_t split_stride = (size_t)sum.vpad * sum.rows_padded;
  float part0[IN_FLIGHT], part1[IN_FLIGHT], in0[HEADS], in1[HEADS];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int u = 0; u < IN_FLIGHT; ++u)
      if (s0 + u < sum.splits) {
        part0[u] = partials[(size_t)(s0 + u) * split_stride + i0];
        part1[u] = partials[(size_t)(s0 + u) * split_stride + i1];
      }
  };
  if (summing) fetch(0);
#pragma unroll
  for (int h = 0; h < HEADS; ++h) {
    in0[h] = in1[h] = 0.f;
    if (!summing && live && head0 + h * GROUPS < heads) {
      const float* src = qkv + (row * heads + head0 + h * GROUPS) * D;
      in0[h] = src[i0];
      in1[h] = src[i1];
    }
  }
  double s = 0.0, c = 1.0;
  if (group == 0 && (int)blockIdx.x * HEADS * GROUPS < q_heads + pool.kv_heads) sincos((double)pos * freq, &s, &c);
  if (GROUPS > 1) {
    if (group == 0 && live) angle[j] = make_double2(s, c);
    __syncthreads();
    s = angle[j].x;
    c = angle[j].y;
  }
  if (summing) {
    for (int s0 = 0; s0 < sum.splits; s0 += IN_FLIGHT) {
      if (s0 > 0) fetch(s0);
#pragma unroll
      for (int u = 0; u < IN_FLIGHT; ++u)
        if (s0 + u < sum.splits && live) {
          in0[0] += part0[u];
          in1[0] += part1[u];
        }
    }
  }
#pragma unroll
  for (int h = 0; h < HEADS; ++h) {
    const int head = head0 + h * GROUPS;
    const bool is_q = head < q_heads, is_k = !is_q && head < q_heads + pool.kv_heads;
    float r0 = in0[h], r1 = in1[h];
    if (is_q || is_k) {
      const double first = (double)r0, second = (double)r1;
      r0 = (float)__dsub_rn(__dmul_rn(first, c), __dmul_rn(second, s));
      r1 = (float)__dadd_rn(__dmul_rn(second, c), __dmul_rn(first, s));
    }
    if (is_q) {
      float* dst = q_out + (row * q_heads + head) * D;
      if (live) {
        dst[i0] = r0;
        dst[i1] = r1;
      }
    }
    const bool cached = !is_q && head < heads && info.advance > 0;  // a padded lane caches nothing
    const int kv_head = is_k ? head - q_heads : head - q_heads - pool.kv_heads;
    const size_t dst = cached ? pool_elem(pool, page, kv_head, slot) : 0;
    void* slab = is_k ? pool.k : pool.v;
    if (pool.dtype == kKvU8) {
      // the int8 tier: one scale per cached row, as kv_append_kernel (pool.rs:224-240)
      if (HEADS * GROUPS == 1 && !cached) return;  // the same for the whole CTA; with more heads all threads meet at the barriers
      float amax = fmaxf(fabsf(r0), fabsf(r1));
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
      if (h > 0) __syncthreads();  // the previous head's maxima have been read
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
      __syncthreads();
      if (!cached) continue;
      amax = 0.0f;
      for (int w = group * (width >> 5); w < (group + 1) * (width >> 5); ++w) amax = fmaxf(amax, red[w]);
      const float scale = __fadd_rn(__fdiv_rn(amax, 127.0f), 1e-12f);
      if (pair == 0) (is_k ? pool.k_scale : pool.v_scale)[pool_scale_index(pool, page, kv_head, slot)] = scale;
      const float c0 = fminf(fmaxf(roundf(__fdiv_rn(r0, scale)), -127.0f), 127.0f) + 128.0f;
      const float c1 = fminf(fmaxf(roundf(__fdiv_rn(r1, scale)), -127.0f), 127.0f) + 128.0f;
      if (live) {
        reinterpret_cast<uint8_t*>(slab)[dst + i0] = (uint8_t)c0;
        reinterpret_cast<uint8_t*>(slab)[dst + i1] = (uint8_t)c1;
      }
      continue;
    }
    if (!live || !cached) continue;
    pool_store(pool, slab, dst + i0, r0);
    pool_store(pool, slab, dst + i1, r1);
  }
}

cudaError_t launch_rope_append(const PoolView& pool, const float* qkv, const LaneInfo* lanes, const int* tables,
                               const double* inv_freq, int layout, int batch, int q_heads, float* q_out,
                               cudaStream_t stream, const DeferredSum* sum, int tokens) {
  if (batch == 0) return cudaSuccess;
  const int heads = q_heads + 2 * pool.kv_heads, width = std::max(32, (pool.head_dim / 2 + 31) / 32 * 32);
  // several heads per CTA once the rows alone fill the SMs; the sums of split projections are only taken head by head
  const bool many = (int64_t)batch * tokens >= 128 && !(sum && sum->splits > 0) && width <= 64;
  const int per = many ? 16 : 1;
  const dim3 grid((unsigned)((heads + per - 1) / per), (unsigned)batch, (unsigned)tokens);
  return launch_chained(many ? rope_append_kernel<4, 4> : rope_append_kernel<1, 1>, grid, dim3((unsigned)(many ? 4 * width : width)), 0, stream, pool, qkv, lanes,
                        tables, inv_freq, layout, q_heads, q_out, sum ? *sum : DeferredSum());
}

__global__ void record_step_kernel(const uint32_t* tokens, uint32_t* ids,
                                   uint32_t* history, int* step_counter, LaneInfo* lanes, int batch,
                                   long long window) {
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  const int step = *step_counter;
  for (int i = threadIdx.x; i < batch; i += blockDim.x) {
    const uint32_t tok = tokens[i];
    ids[i] = tok;
    history[(size_t)step * batch + i] = tok;
    if (lanes[i].advance > 0) {
      lanes[i].cursor += 1;
      if (window >= 0) lanes[i].start = (int)max((long long)lanes[i].cursor + 1 - window, 0ll);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *step_counter = step + 1;
}
cudaError_t launch_record_step(const uint32_t* tokens, uint32_t* ids, uint32_t* history, int* step_counter, LaneInfo* lanes,
                               int batch, long long window, cudaStream_t stream) {
  return launch_chained(record_step_kernel, dim3(1), dim3(128), 0, stream, tokens, ids, history, step_counter, lanes, batch, window);
}

// Debug/test read-back of logical token rows (row = block*block_size + offset) as f32
// [n, kv_heads*head_dim] in the reference's row order, dequantised for the u8 tier.
__global__ void pool_read_rows_kernel(PoolView pool, const uint32_t* __restrict__ rows, int64_t n, float* __restrict__ out,
                                      int which) {
  const int64_t width = (int64_t)pool.kv_heads * pool.head_dim;
  const int64_t total = n * width;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / width, e = idx - i * width;
    const int head = (int)(e / pool.head_dim), d = (int)(e % pool.head_dim);
    const int page = (int)(rows[i] / pool.block_size), slot = (int)(rows[i] % pool.block_size);
    out[idx] = pool_load(pool, which == 0 ? pool.k : pool.v, which == 0 ? pool.k_scale : pool.v_scale,
                         pool_elem(pool, page, head, slot) + d, pool_scale_index(pool, page, head, slot));
  }
}
cudaError_t launch_pool_read_rows(const PoolView& pool, const uint32_t* rows, int64_t n, float* out, int which,
                                  cudaStream_t stream) {
  const int64_t total = n * pool.kv_heads * pool.head_dim;
  if (total == 0) return cudaSuccess;
  pool_read_rows_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256, 148 * 8), 256, 0, stream>>>(pool, rows, n, out, which);
  return cudaGetLastError();
}

}  // namespace etc
