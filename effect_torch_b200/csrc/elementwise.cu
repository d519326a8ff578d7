// Dense and elementwise kernels of the decode graph for sm_100a: exact-order dense linear,
// RMSNorm, RoPE, SwiGLU, residual add, greedy argmax, dense embedding gather and the layout
// shuffles around attention. All are HBM/latency-bound single-pass kernels.
//
// Replaces, for the CUDA backend: crates/runtime-cpu/src/matmul.rs:192-231 (naive_into),
// crates/runtime-cpu/src/composed.rs:1457-1487 (rms_norm_forward_into_impl) and :2683-2729
// (rotary_forward_into_impl), the FusedElementwise regions evaluating
// packages/core/src/Tensor.ts:1240-1245,1537-1540 (sigmoid/silu), and the greedy branch of
// crates/runtime/src/sampling.rs:88-105.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "activation.cuh"
#include "chain.cuh"
#include "kernels.h"

namespace etc {

// silu(gate) * up as the reference's expression interpreter evaluates it, see swiglu_kernel.
__device__ __forceinline__ float swiglu_value(float g, float up, int exact) {
  if (!exact) return __fmul_rn(silu_tanh(g), up);
  const float th = (float)tanh((double)(g * 0.5f));
  return __fmul_rn(__fmul_rn(g, __fadd_rn(th * 0.5f, 0.5f)), up);
}

__device__ __forceinline__ double square4(const float4& v) {
  return (double)v.x * (double)v.x + (double)v.y * (double)v.y + (double)v.z * (double)v.z + (double)v.w * (double)v.w;
}
__device__ __forceinline__ float4 scale4(const float4& v, double scale, const float4& w) {
  return make_float4((float)__dmul_rn(__dmul_rn((double)v.x, scale), (double)w.x), (float)__dmul_rn(__dmul_rn((double)v.y, scale), (double)w.y),
                     (float)__dmul_rn(__dmul_rn((double)v.z, scale), (double)w.z), (float)__dmul_rn(__dmul_rn((double)v.w, scale), (double)w.w));
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

constexpr int kNormThreads = 256, kNormItems = 8192 / 4 / kNormThreads;

// --------------------------------------------------------------------------------------------
// Dense linear, bit-exact with the reference: every output element is one sequential fmaf chain over k
// (out = fma(x[m,k], W[n,k], out)), four cycles per k whatever is done, so for the small models that run in f32 what counts is
// that nothing else adds to the chain: a ring of four 64-column stages filled by cp.async (one exposed load latency per
// launch instead of one per 32 columns), 16-byte shared-memory reads (rows padded to 272 bytes: conflict free), launches
// chained, and up to three weights per launch (q, k and v side by side in one output; gate and up with the SwiGLU between
// them; the residual added on the way out). A CTA computes 32 outputs x 8 * MT input rows; MT = 4 reuses a weight read for
// four rows' chains where there are that many.
// --------------------------------------------------------------------------------------------
constexpr int kDenseK = 64, kDenseStages = 4, kDensePad = kDenseK + 4;

template <int MT, bool SWIGLU>
struct DenseCfg {
  static constexpr int kRowsW = 32 * (SWIGLU ? 2 : 1), kRowsX = 8 * MT;
  static constexpr int kStageFloats = (kRowsW + kRowsX) * kDensePad;
  static constexpr size_t kSmemBytes = (size_t)kDenseStages * kStageFloats * sizeof(float);
};

template <int MT, bool SWIGLU>
__global__ void __launch_bounds__(256) dense_linear_kernel(DenseArgs a) {
  using Cfg = DenseCfg<MT, SWIGLU>;
  chain_release();
  extern __shared__ __align__(16) float ring[];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // output within the tile, input row within the tile
  int tile = blockIdx.x, part = 0;
  if (!SWIGLU)
    while (part + 1 < a.parts && tile >= (int)((a.n[part] + 31) / 32)) tile -= (int)((a.n[part++] + 31) / 32);
  const int64_t n = a.n[part], n0 = (int64_t)tile * 32, m0 = (int64_t)blockIdx.y * Cfg::kRowsX;
  const int k = (int)a.k, chunks = (k + kDenseK - 1) / kDenseK;
  // rows beyond the matrix repeat its last one: their results are not stored
  auto fill = [&](int chunk, bool weights, bool inputs) {
    float* stage = ring + (chunk % kDenseStages) * Cfg::kStageFloats;
    for (int i = threadIdx.x; i < (Cfg::kRowsW + Cfg::kRowsX) * (kDenseK / 4); i += 256) {
      const int row = i / (kDenseK / 4), c = chunk * kDenseK + 4 * (i % (kDenseK / 4));
      const bool is_w = row < Cfg::kRowsW;
      if (c >= k || !(is_w ? weights : inputs)) continue;
      const float* src = is_w ? a.w[SWIGLU ? row / 32 : part] + min(n0 + row % 32, n - 1) * k + c : a.x + min(m0 + row - Cfg::kRowsW, a.m - 1) * k + c;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(stage + row * kDensePad + 4 * (i % (kDenseK / 4)));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  // the first stages' weights depend on no earlier kernel of the decoder's step (a.constant_weights)
  if (a.constant_weights)
    for (int c = 0; c < kDenseStages - 1; ++c) fill(c, c < chunks, false);
  chain_wait();
  for (int c = 0; c < kDenseStages - 1; ++c) {
    fill(c, c < chunks && !a.constant_weights, c < chunks);
    commit();
  }
  float acc[MT] = {}, up[MT] = {};
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kDenseStages - 2) : "memory");
    __syncthreads();
    if (c + kDenseStages - 1 < chunks) fill(c + kDenseStages - 1, true, true);
    commit();
    const float* stage = ring + (c % kDenseStages) * Cfg::kStageFloats;
    const int len = min(kDenseK, k - c * kDenseK);
#pragma unroll 4
    for (int kk = 0; kk < len; kk += 4) {
      const float4 w = *reinterpret_cast<const float4*>(stage + tx * kDensePad + kk);
      float4 w2;
      if (SWIGLU) w2 = *reinterpret_cast<const float4*>(stage + (32 + tx) * kDensePad + kk);
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        const float4 x = *reinterpret_cast<const float4*>(stage + (Cfg::kRowsW + ty + 8 * t) * kDensePad + kk);
        acc[t] = fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, acc[t]))));
        if (SWIGLU) up[t] = fmaf(x.w, w2.w, fmaf(x.z, w2.z, fmaf(x.y, w2.y, fmaf(x.x, w2.x, up[t]))));
      }
    }
  }
  const int64_t col = n0 + tx;
  if (col >= n) return;
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    const int64_t row = m0 + ty + 8 * t;
    if (row >= a.m) break;
    const int64_t at = row * a.out_stride + col;
    if (SWIGLU) {
      a.out[0][at] = swiglu_value(acc[t], up[t], a.exact);
    } else {
      const float v = a.bias ? acc[t] + a.bias[col] : acc[t];
      a.out[part][at] = a.residual ? __fadd_rn(a.residual[at], v) : v;
    }
  }
}

// The same chain where a decode step's few rows meet a narrow weight (the small f32 models): a CTA holds the whole of 32 weight
// rows in shared memory, fetched before the wait for the kernel ahead, so that only the input rows, the chain itself and the
// store are left behind it. A warp carries ROWS input rows. (In the ring above eight warps read the same tile, 10 cycles of
// shared-memory path per k where the chain needs four, with a barrier per 64 columns: 4 rows in a step's chain took 9 us for
// k = 688 and 4.1 for 256, now 3.8 and 2.2.) The norm ahead of the projection may come along where that pays (dense_norm_rides): every
// CTA computes it for its own copy of the rows, with the sums of rmsnorm_rows_kernel, instead of a launch.
// With SWIGLU lanes 0 to 15 hold gate rows and lanes 16 to 31 their up rows.
constexpr int kNarrowThreads = 128, kNarrowRows = 16;
constexpr size_t kNarrowSmem = 220 * 1024;
static size_t narrow_smem(const DenseArgs& a) { return sizeof(float) * (32 * (size_t)(a.k + 4) + (size_t)a.m * a.k); }

template <int ROWS, bool SWIGLU>
__global__ void __launch_bounds__(kNarrowThreads) dense_narrow_kernel(DenseArgs a) {
  chain_release();
  extern __shared__ __align__(16) float tile_s[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int OUTS = SWIGLU ? 16 : 32;
  int tile = blockIdx.x, part = 0;
  if (!SWIGLU)
    while (part + 1 < a.parts && tile >= (int)((a.n[part] + 31) / 32)) tile -= (int)((a.n[part++] + 31) / 32);
  const int64_t n = a.n[part], n0 = (int64_t)tile * OUTS;
  const int k = (int)a.k, quads = k / 4, pitch = k + 4, m = (int)a.m;
  float* x_s = tile_s + 32 * pitch;
  auto copy16 = [](float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
  };
  auto fill_weights = [&] {  // rows beyond the matrix repeat its last one: their results are not stored
    for (int r = warp; r < 32; r += kNarrowThreads / 32) {
      const float* src = (SWIGLU ? a.w[r / OUTS] : a.w[part]) + min(n0 + r % OUTS, n - 1) * k;
      for (int q = lane; q < quads; q += 32) copy16(tile_s + r * pitch + 4 * q, src + 4 * q);
    }
  };
  if (a.constant_weights) fill_weights();
  chain_wait();
  if (!a.constant_weights) fill_weights();
  if (a.norm_weight) {
    for (int r = warp; r < m; r += kNarrowThreads / 32) {
      const float4* src = reinterpret_cast<const float4*>(a.x + (int64_t)r * k);
      float4* dst = reinterpret_cast<float4*>(x_s + r * k);
      double total = 0.0;
      for (int p = 0; p < kNormThreads / 32 && 32 * p < quads; ++p) {  // the partial sum of warp p of rmsnorm_rows_kernel
        double sum = 0.0;
        for (int q = 32 * p + lane; q < quads; q += kNormThreads) {
          const float4 v = src[q];
          dst[q] = v;
          sum += square4(v);
        }
        total += warp_sum(sum);
      }
      const double scale = 1.0 / sqrt(total / (double)k + a.norm_eps);
      for (int q = lane; q < quads; q += 32) dst[q] = scale4(dst[q], scale, reinterpret_cast<const float4*>(a.norm_weight)[q]);
    }
  } else {
    for (int i = threadIdx.x; i < m * quads; i += kNarrowThreads) copy16(x_s + 4 * i, a.x + 4 * (int64_t)i);
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int row0 = warp * ROWS;
  if (row0 >= m) return;
  const float4* w4 = reinterpret_cast<const float4*>(tile_s + lane * pitch);
  const float4* x4[ROWS];
  float acc[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    x4[r] = reinterpret_cast<const float4*>(x_s + min(row0 + r, m - 1) * k);
    acc[r] = 0.0f;
  }
  // a few quads at a time, the next ones on their way while these are added
  constexpr int AHEAD = ROWS == 4 ? 2 : 4;
  float4 w[2][AHEAD], x[2][AHEAD][ROWS];
  auto fetch = [&](int buffer, int q0) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int q = min(q0 + u, quads - 1);
      w[buffer][u] = w4[q];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) x[buffer][u][r] = x4[r][q];
    }
  };
  auto add = [&](int buffer, int n_quads) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (u >= n_quads) break;
      const float4 wv = w[buffer][u];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float4 xv = x[buffer][u][r];
        acc[r] = fmaf(xv.w, wv.w, fmaf(xv.z, wv.z, fmaf(xv.y, wv.y, fmaf(xv.x, wv.x, acc[r]))));
      }
    }
  };
  fetch(0, 0);
  int q = 0;
  for (; q + 2 * AHEAD <= quads; q += 2 * AHEAD) {
    fetch(1, q + AHEAD);
    add(0, AHEAD);
    fetch(0, q + 2 * AHEAD);
    add(1, AHEAD);
  }
  if (q < quads) {
    fetch(1, q + AHEAD);
    add(0, min(AHEAD, quads - q));
    add(1, quads - q - AHEAD);
  }
  const int64_t col = n0 + lane % OUTS;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    float value = acc[r];
    if (SWIGLU) value = swiglu_value(value, __shfl_down_sync(0xffffffffu, value, 16), a.exact);
    if (row0 + r >= m || col >= n || lane >= OUTS) continue;
    const int64_t at = (row0 + r) * a.out_stride + col;
    if (!SWIGLU && a.bias) value += a.bias[col];
    if (!SWIGLU && a.residual) value = __fadd_rn(a.residual[at], value);
    a.out[part][at] = value;
  }
}

// The same chain for operands that 16-byte copies cannot fetch (k not a multiple of 4, unaligned pointers).
__global__ void __launch_bounds__(256) linear_f32_kernel(const float* __restrict__ x, int64_t m, int64_t k,
                                                         const float* __restrict__ w, int64_t n,
                                                         const float* __restrict__ bias, const float* residual, float* out, int64_t out_stride) {
  __shared__ float ws[32][33];
  __shared__ float xs[8][32];
  const int tx = threadIdx.x, ty = threadIdx.y;  // tx: output column within tile, ty: input row within tile
  const int64_t n0 = (int64_t)blockIdx.x * 32, m0 = (int64_t)blockIdx.y * 8;
  float acc = 0.0f;
  for (int64_t k0 = 0; k0 < k; k0 += 32) {
    // W tile: rows n0..n0+31, columns k0..k0+31 (coalesced along k)
    for (int r = ty; r < 32; r += 8) {
      const int64_t nn = n0 + r, kk = k0 + tx;
      ws[r][tx] = (nn < n && kk < k) ? w[nn * k + kk] : 0.0f;
    }
    {
      const int64_t mm = m0 + ty, kk = k0 + tx;
      xs[ty][tx] = (mm < m && kk < k) ? x[mm * k + kk] : 0.0f;
    }
    __syncthreads();
    const int len = (int)min((int64_t)32, k - k0);
    for (int kk = 0; kk < len; ++kk) acc = fmaf(xs[ty][kk], ws[tx][kk], acc);
    __syncthreads();
  }
  const int64_t mm = m0 + ty, nn = n0 + tx;
  if (mm < m && nn < n) {
    const float v = bias ? acc + bias[nn] : acc;
    out[mm * out_stride + nn] = residual ? __fadd_rn(residual[mm * out_stride + nn], v) : v;
  }
}

bool dense_linear_supported(const DenseArgs& a) {
  if (a.k <= 0 || a.k % 4 != 0 || a.k > INT32_MAX || ((uintptr_t)a.x % 16) != 0) return false;
  for (const float* w : a.w)
    if (((uintptr_t)w % 16) != 0) return false;
  return true;
}

template <int MT, bool SWIGLU>
static cudaError_t launch_dense_t(const DenseArgs& a, cudaStream_t stream) {
  constexpr size_t smem = DenseCfg<MT, SWIGLU>::kSmemBytes;
  auto kernel = dense_linear_kernel<MT, SWIGLU>;
  const cudaError_t attr = opt_in_shared_memory(kernel, smem);
  if (attr != cudaSuccess) return attr;
  unsigned tiles = 0;
  for (int p = 0; p < (SWIGLU ? 1 : a.parts); ++p) tiles += (unsigned)((a.n[p] + 31) / 32);
  return launch_chained(kernel, dim3(tiles, (unsigned)((a.m + 8 * MT - 1) / (8 * MT))), dim3(256), smem, stream, a);
}

static unsigned narrow_tiles(const DenseArgs& a) {
  unsigned tiles = 0;
  for (int p = 0; p < (a.swiglu ? 1 : a.parts); ++p) tiles += (unsigned)((a.n[p] + (a.swiglu ? 15 : 31)) / (a.swiglu ? 16 : 32));
  return tiles;
}
// Five to eight rows fill the ring's CTAs, whose copies overlap its chains; here one CTA to an SM loads and then computes, and after
// some waves of that the ring is ahead. [n x k] x rows, this kernel and the ring: [40000 x 728] x 8 57.9 and 50.7 us, [65536 x 800] x 7
// 92.7 and 84.4, [128256 x 1024] x 8 220 and 207; x 5 [65536 x 1024] 110 and 114, [128256 x 800] 177 and 165. Up to four rows
// and from nine on, where the ring's rows are not full or are read twice, this kernel is 1.15 to 5 times as fast at every width.
static bool ring_is_faster(const DenseArgs& a) {
  const bool alone = 2 * (narrow_smem(a) + kCtaSharedReserve) > kSmSharedBytes;
  return !a.swiglu && alone && a.m > 4 && a.m <= 8 && narrow_tiles(a) > (a.m <= 6 ? 16u : 8u) * (unsigned)a.sm_count;
}
bool dense_narrow_supported(const DenseArgs& a) {
  return dense_linear_supported(a) && a.m <= kNarrowRows && narrow_smem(a) <= kNarrowSmem && ((uintptr_t)a.norm_weight % 16) == 0 && !ring_is_faster(a);
}

// The norm inside saves a launch, of which the chain hides all but a few tenths of a microsecond, and costs every CTA its rows' sums
// one after the other. It pays with a row per warp, two 16-byte loads per lane and row, and one CTA per SM. Steps of four layers, inside
// and as launches: 256 columns x 1 row 74.2 and 75.8 us, x 4 82.4 and 82.9; beyond the line 256 x 5 102 and 97, x 16 158 and
// 127, 512 x 1 115.5 and 114.3, 512 x 8 197 and 170, 1280 x 8 (128256 outputs) 1143 and 638.
bool dense_norm_rides(const DenseArgs& a, int64_t tiles) {
  return dense_narrow_supported(a) && a.m <= 4 && a.k <= 256 && tiles <= a.sm_count;
}

template <bool SWIGLU>
static cudaError_t launch_narrow(const DenseArgs& a, cudaStream_t stream) {
  // Four warps, one per scheduler: a 16-byte load takes eight cycles of a scheduler's register path, be it a broadcast input or
  // a weight, so that a row per warp (two loads to 16 cycles of chained FMAs) does better than two rows in each of two warps.
  auto kernel = a.m <= 4 ? dense_narrow_kernel<1, SWIGLU> : a.m <= 8 ? dense_narrow_kernel<2, SWIGLU> : dense_narrow_kernel<4, SWIGLU>;
  const cudaError_t attr = opt_in_shared_memory(kernel, kNarrowSmem);
  if (attr != cudaSuccess) return attr;
  return launch_chained(kernel, dim3(narrow_tiles(a)), dim3(kNarrowThreads), narrow_smem(a), stream, a);
}

cudaError_t launch_dense_linear(const DenseArgs& a, cudaStream_t stream) {
  if (a.m == 0 || a.n[0] == 0) return cudaSuccess;
  if (dense_narrow_supported(a)) return a.swiglu ? launch_narrow<true>(a, stream) : launch_narrow<false>(a, stream);
  if (a.norm_weight) return cudaErrorInvalidValue;
  if (!dense_linear_supported(a)) {
    if (a.swiglu) return cudaErrorInvalidValue;
    for (int p = 0; p < a.parts; ++p) {
      const dim3 grid((unsigned)((a.n[p] + 31) / 32), (unsigned)((a.m + 7) / 8));
      linear_f32_kernel<<<grid, dim3(32, 8), 0, stream>>>(a.x, a.m, a.k, a.w[p], a.n[p], a.bias, a.residual, a.out[p], a.out_stride);
    }
    return cudaGetLastError();
  }
  if (a.m > 16) return a.swiglu ? launch_dense_t<4, true>(a, stream) : launch_dense_t<4, false>(a, stream);
  return a.swiglu ? launch_dense_t<1, true>(a, stream) : launch_dense_t<1, false>(a, stream);
}

cudaError_t launch_linear_f32(const float* x, int64_t m, int64_t k, const float* w, int64_t n, const float* bias,
                              float* out, int sm_count, cudaStream_t stream) {
  DenseArgs a;
  a.sm_count = sm_count;
  a.x = x; a.m = m; a.k = k; a.w[0] = w; a.n[0] = n; a.out[0] = out; a.out_stride = n; a.bias = bias;
  return launch_dense_linear(a, stream);
}

// --------------------------------------------------------------------------------------------
// RMSNorm: one CTA per row, sum of squares and the scaling in f64 like the reference
// (scale = 1/sqrt(ms/n + eps); out = f32(x * scale * w)). The f64 block reduction is a tree, so
// the sum can differ from the reference's sequential sum in the last f64 bits only.
// --------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ weight,
                                                      double eps, int64_t n, float* __restrict__ out) {
  __shared__ double partial[8];
  __shared__ double scale_s;
  const float* src = x + (int64_t)blockIdx.x * n;
  double sum = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = (double)src[i];
    sum += v * v;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) total += partial[i];
    scale_s = 1.0 / sqrt(total / (double)n + eps);
  }
  __syncthreads();
  const double scale = scale_s;
  float* dst = out + (int64_t)blockIdx.x * n;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double w = weight ? (double)weight[i] : 1.0;
    dst[i] = (float)(__dmul_rn(__dmul_rn((double)src[i], scale), w));
  }
}

// Single-pass variants for n <= 8192, n % 4 == 0: the row stays in registers between the reduction and the scaling (same
// f64 arithmetic). f32 row-major:
__global__ void __launch_bounds__(kNormThreads) rmsnorm_rows_kernel(const float* x, const float* weight, double eps, int n,
                                                                   float* out) {
  __shared__ double partial[kNormThreads / 32];
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  const int chunks = n / 4;
  const float4* src = reinterpret_cast<const float4*>(x + (size_t)blockIdx.x * n);
  float4 v[kNormItems];
  double sum = 0.0;
#pragma unroll
  for (int j = 0; j < kNormItems; ++j) {
    const int c = threadIdx.x + kNormThreads * j;
    v[j] = c < chunks ? src[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    sum += square4(v[j]);
  }
  sum = warp_sum(sum);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = sum;
  __syncthreads();
  double total = 0.0;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) total += partial[i];
  const double scale = 1.0 / sqrt(total / (double)n + eps);
#pragma unroll
  for (int j = 0; j < kNormItems; ++j) {
    const int c = threadIdx.x + kNormThreads * j;
    if (c >= chunks) continue;
    const float4 w = weight ? reinterpret_cast<const float4*>(weight)[c] : make_float4(1.f, 1.f, 1.f, 1.f);
    reinterpret_cast<float4*>(out + (size_t)blockIdx.x * n)[c] = scale4(v[j], scale, w);
  }
}

// The same for a few rows into the f16 hand-off layout, first adding a projection's split-K partials (in split order) onto
// the row and storing it back: the residual update that the projection's own sum kernel would have done. sum_in.splits may
// be 0: the row as it is.
//
// Bound by latency: a row and its partials (up to 10 x 32 KB) come from L2, and every kernel of a decode step waits for this
// one. A cluster of four CTAs shares a row, so that the partials come through four SMs; each thread has its loads of ten
// splits in flight at once, and the warps' sums of squares are exchanged through distributed shared memory. One CTA per row
// with four loads in flight took 7.5 us for 32 rows of 4096 with 9 splits.
constexpr int kNormCluster = 4;
__global__ void __launch_bounds__(kNormThreads) sum_rmsnorm_xh_kernel(float* x, const float* __restrict__ weight, double eps, int n, __half* out_xh,
                                                                     int xh_nv, DeferredSum sum_in) {
  namespace cg = cooperative_groups;
  constexpr int ITEMS = kNormItems / kNormCluster, WARPS = kNormThreads / 32;
  static_assert(kNormCluster * WARPS == 32, "one sum per lane");
  __shared__ double partial[32];
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // waited for below: the peers' shared memory exists
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  const int chunks = n / 4, first = blockIdx.x * kNormThreads + threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // launched by the decoder alone, whose norm weights no kernel writes after the load: they are fetched while the kernel
  // before this one is still running
  float4 w[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int c = first + kNormCluster * kNormThreads * j;
    w[j] = weight && c < chunks ? reinterpret_cast<const float4*>(weight)[c] : make_float4(1.f, 1.f, 1.f, 1.f);
  }
  chain_wait();
  const int row = blockIdx.y;
  float4* src = reinterpret_cast<float4*>(x + (size_t)row * n);
  float4 v[ITEMS];
  double sum = 0.0;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int c = first + kNormCluster * kNormThreads * j;
    v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c >= chunks) continue;
    v[j] = src[c];
    if (sum_in.splits > 0) {
      constexpr int IN_FLIGHT = 10;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      const float* base = sum_in.partials + (size_t)row * sum_in.rows_padded + 4 * c;
      const size_t split_stride = (size_t)sum_in.vpad * sum_in.rows_padded;
      for (int s0 = 0; s0 < sum_in.splits; s0 += IN_FLIGHT) {
        float4 p[IN_FLIGHT];
#pragma unroll
        for (int u = 0; u < IN_FLIGHT; ++u)
          if (s0 + u < sum_in.splits) p[u] = *reinterpret_cast<const float4*>(base + (size_t)(s0 + u) * split_stride);
#pragma unroll
        for (int u = 0; u < IN_FLIGHT; ++u)
          if (s0 + u < sum_in.splits) { acc.x += p[u].x; acc.y += p[u].y; acc.z += p[u].z; acc.w += p[u].w; }
      }
      v[j].x += acc.x; v[j].y += acc.y; v[j].z += acc.z; v[j].w += acc.w;
    }
    sum += square4(v[j]);
  }
  if (sum_in.splits > 0) {
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      if (first + kNormCluster * kNormThreads * j < chunks) src[first + kNormCluster * kNormThreads * j] = v[j];
  }
  sum = warp_sum(sum);
  cluster.barrier_wait();
  if (lane < kNormCluster) cluster.map_shared_rank(partial, lane)[blockIdx.x * WARPS + warp] = sum;
  cluster.sync();
  const double scale = 1.0 / sqrt(warp_sum(partial[lane]) / (double)n + eps);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int c = first + kNormCluster * kNormThreads * j;
    if (c < chunks) *reinterpret_cast<uint2*>(out_xh + hand_off_cell(c >> 1, row, xh_nv, n / 8) + 4 * (c & 1)) = pack4(scale4(v[j], scale, w[j]));
  }
}

// The same for many rows (hand-off chunks of 128), without partials. A CTA takes two neighbouring rows: two lanes exchange
// halves, so that each stores 16 bytes and the pair fills a sector of the hand-off layout. With one row per CTA and stores of
// 8 bytes that each touch a sector of their own, 2048 rows of 4096 took 32 us.
template <int ITEMS>
__global__ void __launch_bounds__(kNormThreads) rmsnorm_chunk_xh_kernel(const float* x, const float* __restrict__ weight, double eps, int rows, int n,
                                                                       __half* out_xh) {
  __shared__ double partial[2][kNormThreads / 32];
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  const int chunks = n / 4, row0 = 2 * blockIdx.x;
  const bool both = row0 + 1 < rows;
  const float4* src0 = reinterpret_cast<const float4*>(x + (size_t)row0 * n);
  const float4* src1 = both ? src0 + chunks : src0;
  float4 v0[ITEMS], v1[ITEMS];
  double sum0 = 0.0, sum1 = 0.0;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int c = threadIdx.x + kNormThreads * j;
    v0[j] = c < chunks ? src0[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    v1[j] = c < chunks ? src1[c] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    sum0 += square4(v0[j]);
    sum1 += square4(v1[j]);
  }
  sum0 = warp_sum(sum0);
  sum1 = warp_sum(sum1);
  if ((threadIdx.x & 31) == 0) {
    partial[0][threadIdx.x >> 5] = sum0;
    partial[1][threadIdx.x >> 5] = sum1;
  }
  __syncthreads();
  sum0 = sum1 = 0.0;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) {
    sum0 += partial[0][i];
    sum1 += partial[1][i];
  }
  const double scale0 = 1.0 / sqrt(sum0 / (double)n + eps), scale1 = 1.0 / sqrt(sum1 / (double)n + eps);
  const bool odd = threadIdx.x & 1;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int c = threadIdx.x + kNormThreads * j;
    const float4 w = weight && c < chunks ? reinterpret_cast<const float4*>(weight)[c] : make_float4(1.f, 1.f, 1.f, 1.f);
    const uint2 a = pack4(scale4(v0[j], scale0, w)), b = pack4(scale4(v1[j], scale1, w)), give = odd ? a : b;
    const uint2 got = make_uint2(__shfl_xor_sync(0xffffffffu, give.x, 1), __shfl_xor_sync(0xffffffffu, give.y, 1));
    if (c < chunks && (!odd || both))  // n % 8 == 0: both lanes of a pair are inside the row
      *reinterpret_cast<uint4*>(out_xh + hand_off_cell(c >> 1, row0 + odd, 128, n / 8)) =
          odd ? make_uint4(got.x, got.y, b.x, b.y) : make_uint4(a.x, a.y, got.x, got.y);
  }
}

static bool rmsnorm_fast_ok(const float* x, const float* weight, int64_t n) {
  return n % 4 == 0 && n <= 8192 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)weight % 16) == 0;
}

cudaError_t launch_rmsnorm(const float* x, const float* weight, double eps, int64_t rows, int64_t n, float* out,
                           cudaStream_t stream) {
  if (rows == 0) return cudaSuccess;
  if (rmsnorm_fast_ok(x, weight, n) && ((uintptr_t)out % 16) == 0)
    return launch_chained(rmsnorm_rows_kernel, dim3((unsigned)rows), dim3(kNormThreads), 0, stream, x, weight, eps, (int)n, out);
  else
    rmsnorm_kernel<<<(unsigned)rows, 256, 0, stream>>>(x, weight, eps, n, out);
  return cudaGetLastError();
}

cudaError_t launch_sum_rmsnorm_xh8(float* x, const DeferredSum& sum, const float* weight, double eps, int64_t rows, int64_t n,
                                   __half* out_xh, cudaStream_t stream, int xh_nv) {
  if (rows == 0) return cudaSuccess;
  if (rows > xh_nv && xh_nv != 128) return cudaErrorInvalidValue;
  if (n % 8 != 0 || !rmsnorm_fast_ok(x, weight, n)) return cudaErrorInvalidValue;
  if (sum.splits > 0 && (sum.rows_padded % 4 != 0 || rows > sum.vpad)) return cudaErrorInvalidValue;
  if (rows > 128 && sum.splits == 0) {  // two rows per CTA fill half the SMs, and the sums of a cluster cost more than they save
    const auto kernel = n <= 4096 ? rmsnorm_chunk_xh_kernel<kNormItems / 2> : rmsnorm_chunk_xh_kernel<kNormItems>;
    return launch_chained(kernel, dim3((unsigned)((rows + 1) / 2)), dim3(kNormThreads), 0, stream, (const float*)x, weight, eps, (int)rows, (int)n, out_xh);
  }
  return launch_chained_cluster(sum_rmsnorm_xh_kernel, dim3(kNormCluster, (unsigned)rows), dim3(kNormThreads), 0, stream, (unsigned)kNormCluster, x, weight, eps,
                                (int)n, out_xh, xh_nv, sum);
}

// --------------------------------------------------------------------------------------------
// RoPE on [batch, heads, steps, head_dim] with per-lane cursor offsets. inv_freq[j] =
// theta^(-2j/D) is precomputed on the host in f64 with the same pow() the reference calls;
// angle, sin/cos and the rotation are f64, results are rounded to f32 once.
// --------------------------------------------------------------------------------------------
__global__ void rope_kernel(const float* __restrict__ x, const int64_t* __restrict__ offsets, int64_t n_offsets,
                            const double* __restrict__ inv_freq, int layout, int64_t batch, int64_t heads,
                            int64_t steps, int64_t head_dim, float* __restrict__ out) {
  const int64_t half = head_dim / 2;
  const int64_t total = batch * heads * steps * half;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = idx % half;
    const int64_t row_step = idx / half;  // (batch*heads + head)*steps + step
    const int64_t step = row_step % steps;
    const int64_t b = row_step / (steps * heads);
    const int64_t offset = n_offsets == 1 ? offsets[0] : offsets[b];
    const double angle = (double)(offset + step) * inv_freq[j];
    double s, c;
    sincos(angle, &s, &c);
    const int64_t base = row_step * head_dim;
    const int64_t i0 = layout == 0 ? base + j : base + 2 * j;
    const int64_t i1 = layout == 0 ? base + half + j : base + 2 * j + 1;
    const double first = (double)x[i0], second = (double)x[i1];
    out[i0] = (float)__dsub_rn(__dmul_rn(first, c), __dmul_rn(second, s));
    out[i1] = (float)__dadd_rn(__dmul_rn(second, c), __dmul_rn(first, s));
  }
}

cudaError_t launch_rope(const float* x, const int64_t* offsets, int64_t n_offsets, const double* inv_freq, int layout,
                        int64_t batch, int64_t heads, int64_t steps, int64_t head_dim, float* out, cudaStream_t stream) {
  const int64_t total = batch * heads * steps * (head_dim / 2);
  if (total == 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 8);
  rope_kernel<<<grid, 256, 0, stream>>>(x, offsets, n_offsets, inv_freq, layout, batch, heads, steps, head_dim, out);
  return cudaGetLastError();
}

// --------------------------------------------------------------------------------------------
// silu(gate) * up with the reference's definition sigmoid(x) = tanh(x/2)/2 + 1/2, evaluated in
// f32 like the reference's expression interpreter. exact != 0 takes tanh in f64 and rounds, which
// tracks a correctly rounded tanhf more closely than the device tanhf.
// --------------------------------------------------------------------------------------------
__global__ void swiglu_kernel(const float* __restrict__ gate, const float* __restrict__ up, int64_t n,
                              float* __restrict__ out, int exact) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    out[i] = swiglu_value(gate[i], up[i], exact);
  }
}
cudaError_t launch_swiglu(const float* gate, const float* up, int64_t n, float* out, int exact, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8);
  swiglu_kernel<<<grid, 256, 0, stream>>>(gate, up, n, out, exact);
  return cudaGetLastError();
}

__global__ void add_kernel(const float* __restrict__ a, const float* __restrict__ b, int64_t n, float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __fadd_rn(a[i], b[i]);
}
cudaError_t launch_add(const float* a, const float* b, int64_t n, float* out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8);
  add_kernel<<<grid, 256, 0, stream>>>(a, b, n, out);
  return cudaGetLastError();
}

// --------------------------------------------------------------------------------------------
// Greedy argmax per row: the first index of the maximum (strict >, so the lowest index wins
// ties); a non-finite logit raises the status word with its index.
// A row is served by a cluster of up to 8 CTAs: one CTA per row leaves four fifths of the SMs idle at 32 rows and each
// pulls 512 KB (vocab 128256) through one SM, 17 us where eight slices take 6.
// --------------------------------------------------------------------------------------------
constexpr int kArgmaxThreads = 512;
constexpr int kArgmaxSlice = 8192;  // a row is spread over more CTAs until a slice is this short

// `picks` (optional): the row's (best logit bits, index_base + index) pair, for the exchange between the ranks of a
// vocabulary-parallel head. `mirror` (optional): a second copy of the tokens, in page-locked host memory.
__global__ void __launch_bounds__(kArgmaxThreads) argmax_kernel(const float* logits, int64_t vocab, int64_t slice,
                                                                uint32_t* tokens, DeviceStatus* status, uint2* picks,
                                                                uint32_t index_base, uint32_t* mirror) {
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  namespace cg = cooperative_groups;
  constexpr long long kNone = 0x7fffffffffffffffll;
  constexpr int kWarps = kArgmaxThreads / 32;
  struct Best { float value; long long index, bad; };
  __shared__ Best of_warp[kWarps];
  __shared__ Best of_cta;
  cg::cluster_group cluster = cg::this_cluster();
  const int64_t row_index = blockIdx.x / cluster.num_blocks();
  const int64_t begin = min(vocab, (int64_t)cluster.block_rank() * slice), count = min(vocab, begin + slice) - begin;
  const float* row = logits + row_index * vocab + begin;
  Best best = {-INFINITY, kNone, kNone};
  auto take = [&](float v, int64_t i) {
    if (!isfinite(v)) best.bad = min(best.bad, (long long)(begin + i));
    if (v > best.value) { best.value = v; best.index = begin + i; }
  };
  auto merge = [&](const Best& o) {
    if (o.value > best.value || (o.value == best.value && o.index < best.index)) { best.value = o.value; best.index = o.index; }
    best.bad = min(best.bad, o.bad);
  };
  int64_t head = 0;
  if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    // 16-byte loads, four in flight per thread; a thread's indices still ascend, so strict > keeps the lowest index
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const int64_t n4 = count >> 2;
    int64_t i = threadIdx.x;
    for (; i + 3 * kArgmaxThreads < n4; i += 4 * kArgmaxThreads) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = row4[i + u * kArgmaxThreads];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t base = (i + u * kArgmaxThreads) << 2;
        take(v[u].x, base); take(v[u].y, base + 1); take(v[u].z, base + 2); take(v[u].w, base + 3);
      }
    }
    for (; i < n4; i += kArgmaxThreads) {
      const float4 v = row4[i];
      take(v.x, i << 2); take(v.y, (i << 2) + 1); take(v.z, (i << 2) + 2); take(v.w, (i << 2) + 3);
    }
    head = n4 << 2;
  }
  for (int64_t i = head + threadIdx.x; i < count; i += kArgmaxThreads) take(row[i], i);
  auto reduce_warp = [&]() {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      merge({__shfl_xor_sync(0xffffffffu, best.value, off), __shfl_xor_sync(0xffffffffu, best.index, off), __shfl_xor_sync(0xffffffffu, best.bad, off)});
  };
  reduce_warp();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) of_warp[warp] = best;
  __syncthreads();
  if (warp == 0) {
    if (lane < kWarps) best = of_warp[lane];
    reduce_warp();
    if (lane == 0) of_cta = best;
  }
  cluster.sync();
  if (cluster.block_rank() == 0 && threadIdx.x == 0) {
    for (unsigned r = 1; r < cluster.num_blocks(); ++r) merge(*cluster.map_shared_rank(&of_cta, r));
    // a row of only -inf keeps index 0 like the reference's loop would before it errors
    const uint32_t token = index_base + (best.index == kNone ? 0u : (uint32_t)best.index);
    tokens[row_index] = token;
    if (mirror) mirror[row_index] = token;
    if (picks) picks[row_index] = make_uint2(__float_as_uint(best.value), token);
    if (best.bad != kNone && atomicCAS(&status->code, kStatusNone, kStatusNonFiniteLogit) == kStatusNone) {
      status->value = best.bad;
      status->bound = vocab;
    }
  }
  cluster.sync();  // the other CTAs' shared memory lives until it has been read
}
cudaError_t launch_argmax(const float* logits, int64_t rows, int64_t vocab, uint32_t* tokens, DeviceStatus* status,
                          cudaStream_t stream, uint2* picks, uint32_t index_base, uint32_t* mirror) {
  if (rows == 0) return cudaSuccess;
  unsigned ranks = 1;
  while (ranks < 8 && (vocab + ranks - 1) / ranks > kArgmaxSlice) ranks *= 2;
  const int64_t slice = ((vocab + ranks - 1) / ranks + 3) & ~(int64_t)3;
  return launch_chained_cluster(argmax_kernel, dim3((unsigned)rows * ranks), dim3(kArgmaxThreads), 0, stream, ranks, logits, vocab, slice, tokens, status,
                                picks, index_base, mirror);
}

// Dense f32 embedding gather with the same bounds rule as the quantized embedding.
template <typename Index>
__global__ void embedding_f32_kernel(const Index* indexes, int64_t count, const float* __restrict__ table,
                                     int64_t rows, int64_t columns, float* out, DeviceStatus* status) {
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  const int64_t i = blockIdx.y;
  const long long row = (long long)indexes[i];
  if (row < 0 || row >= rows) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && atomicCAS(&status->code, kStatusNone, kStatusIndexOutOfRange) == kStatusNone) {
      status->value = row;
      status->bound = rows;
    }
    return;
  }
  const float* src = table + row * columns;
  float* dst = out + i * columns;
  if ((columns & 3) == 0 && ((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < columns / 4; c += (int64_t)gridDim.x * blockDim.x)
      reinterpret_cast<float4*>(dst)[c] = reinterpret_cast<const float4*>(src)[c];
    return;
  }
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < columns; c += (int64_t)gridDim.x * blockDim.x) dst[c] = src[c];
}
cudaError_t launch_embedding_f32(const void* indexes, int index_is_i64, int64_t count, const float* table, int64_t rows,
                                 int64_t columns, float* out, DeviceStatus* status, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  dim3 grid((unsigned)std::min<int64_t>((columns + 1023) / 1024, 8), (unsigned)count);
  if (index_is_i64)
    return launch_chained(embedding_f32_kernel<long long>, grid, dim3(256), 0, stream, (const long long*)indexes, count, table, rows, columns, out, status);
  return launch_chained(embedding_f32_kernel<unsigned int>, grid, dim3(256), 0, stream, (const unsigned int*)indexes, count, table, rows, columns, out, status);
}

// LastTokenRow (crates/runtime-cpu/src/napi/mod.rs:3053-3075) for every lane at once.
__global__ void last_token_rows_kernel(const float* __restrict__ src, int64_t lanes, int64_t steps, int64_t width,
                                       int64_t advance, float* __restrict__ out) {
  const int64_t total = lanes * width;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t lane = idx / width, c = idx - lane * width;
    out[idx] = src[(lane * steps + (advance - 1)) * width + c];
  }
}
cudaError_t launch_last_token_rows(const float* src, int64_t lanes, int64_t steps, int64_t width, int64_t advance,
                                   float* out, cudaStream_t stream) {
  const int64_t total = lanes * width;
  if (total == 0) return cudaSuccess;
  last_token_rows_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256, 148 * 8), 256, 0, stream>>>(src, lanes, steps, width, advance, out);
  return cudaGetLastError();
}

}  // namespace etc
