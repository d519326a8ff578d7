// Block-quantized weight kernels for sm_100a: dequantise, quantise, the generic (any codec, raw
// GGUF layout) linear, the row-gather embedding, the split-K sum of the tcgen05 linear and the
// front end that routes a tiled linear to the streaming kernel (qlinear_stream.cu, up to 128 vectors) or to the
// large-batch one (qlinear_umma.cu).
//
// Replaces crates/runtime-cpu/src/quantized.rs (decode_block :90, linear_into :419,
// embedding_into :546) of the reference for the CUDA backend.
#include <cuda_fp16.h>

#include <algorithm>

#include "activation.cuh"
#include "chain.cuh"
#include "codecs.cuh"
#include "kernels.h"

namespace etc {

// ============================================================================================
// Dequantise: bit-exact with the reference decoders. HBM-bound on the f32 output (4 B written per 0.5-1 B read).
// Eight threads share a 256-value window (see Runs in codecs.cuh), so headers and 16-byte payload loads are paid once per
// 32 values; a warp's four windows pass through shared memory because a thread's runs are 64 bytes each and stores that
// far apart would use half of every sector. They leave as 32 bytes per thread (outputs on a 16-byte boundary only: 16). Up to 64
// CTAs per SM, of which some 12 to 16 are resident: a warp waits for its loads before it stores, so what keeps HBM busy is a new
// CTA beside it, not a long loop. [14336 x 4096] (235 MB out) Q4_0 44 us, Q8_0 48; [128256 x 4096] 378 and 414 us, 0.97 of
// the copy bandwidth. 16-byte stores and 12 CTAs per SM: 44, 63, 458 and 551 us; 32-byte stores and 12: 47, 53, 393 and 443.
// One thread per value with byte loads took 170 us on [14336 x 4096] Q4_0.
// ============================================================================================
constexpr int kDequantWarps = 4;

// Eight consecutive values to a 32-byte boundary in one request.
__device__ __forceinline__ void store_eight(float* dst, float4 a, float4 b) {
  asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x),
               "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

template <int CODEC, bool WIDE>
__global__ void __launch_bounds__(kDequantWarps * 32) dequantize_kernel(const uint8_t* __restrict__ packed, int64_t total,
                                                                         float* __restrict__ out) {
  // quads of four values; quad q of a warp's 256 sits at q ^ (bits 2-4 of q's run position) so that neither side conflicts
  __shared__ float4 stage[kDequantWarps][256];
  constexpr int64_t kWindowBytes = 256 / CodecTraits<CODEC>::kValues * CodecTraits<CODEC>::kBytes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, s = lane & 7, w = lane >> 3;
  const int64_t groups = (total + 1023) / 1024;  // of four windows: consecutive values, whatever row they belong to
  const bool widest_out = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
  float4* mine = stage[warp];
  auto place = [](int quad) { return quad ^ ((quad >> 3) & 7); };
  for (int64_t g = blockIdx.x * (int64_t)kDequantWarps + warp; g < groups; g += (int64_t)gridDim.x * kDequantWarps) {
    const int64_t first = g * 1024 + w * 256;
    const bool live = CODEC == kQ4_0 || CODEC == kQ8_0 ? first + s * 32 < total : first < total;
    if (live) {
      const Runs runs = load_runs<CODEC, WIDE>(packed + first / 256 * kWindowBytes, s);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int q0 = (w * 256 + run_column<CODEC>(s, r)) >> 2;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          mine[place(q0 + q)] = make_float4(run_value<CODEC>(runs, r, 4 * q), run_value<CODEC>(runs, r, 4 * q + 1),
                                            run_value<CODEC>(runs, r, 4 * q + 2), run_value<CODEC>(runs, r, 4 * q + 3));
      }
    }
    __syncwarp();
    if (widest_out) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int q = 2 * lane + 64 * j;
        const int64_t at = g * 1024 + 4 * q;
        if (at < total) store_eight(out + at, mine[place(q)], mine[place(q + 1)]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int q = lane + 32 * j;
        const int64_t at = g * 1024 + 4 * q;
        if (at < total) __stcs(reinterpret_cast<float4*>(out + at), mine[place(q)]);
      }
    }
    __syncwarp();
  }
}

// One thread per value, for outputs that are not 16-byte aligned.
template <int CODEC>
__global__ void dequantize_unaligned_kernel(const uint8_t* __restrict__ packed, int64_t total, float* __restrict__ out) {
  constexpr int BV = CodecTraits<CODEC>::kValues, BB = CodecTraits<CODEC>::kBytes;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x)
    out[idx] = decode_elem<CODEC>(packed + idx / BV * BB, (int)(idx % BV));
}

struct DequantLaunch {
  const uint8_t* packed; int64_t rows, columns; float* out; cudaStream_t stream; cudaError_t err;
  template <int CODEC> void operator()() {
    const int64_t total = rows * columns;
    if (total == 0) { err = cudaSuccess; return; }
    if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
      const int64_t blocks = std::min<int64_t>((total + 1024 * kDequantWarps - 1) / (1024 * kDequantWarps), 148 * 64);
      if (kWideBlocks<CODEC> && (reinterpret_cast<uintptr_t>(packed) & 15) == 0)
        dequantize_kernel<CODEC, kWideBlocks<CODEC>><<<(unsigned)blocks, kDequantWarps * 32, 0, stream>>>(packed, total, out);
      else
        dequantize_kernel<CODEC, false><<<(unsigned)blocks, kDequantWarps * 32, 0, stream>>>(packed, total, out);
    } else {
      dequantize_unaligned_kernel<CODEC><<<(unsigned)std::min<int64_t>((total + 255) / 256, 148 * 32), 256, 0, stream>>>(packed, total, out);
    }
    err = cudaGetLastError();
  }
};
cudaError_t launch_dequantize(int codec, const uint8_t* packed, int64_t rows, int64_t columns, float* out,
                              cudaStream_t stream) {
  DequantLaunch l{packed, rows, columns, out, stream, cudaSuccess};
  if (!dispatch_codec(codec, l)) return cudaErrorInvalidValue;
  return l.err;
}

template <int CODEC, typename Index>
__global__ void qembedding_kernel(const Index* __restrict__ indexes, int64_t count, const uint8_t* __restrict__ packed,
                                  int64_t rows, int64_t columns, float* __restrict__ out, DeviceStatus* status) {
  constexpr int BV = CodecTraits<CODEC>::kValues, BB = CodecTraits<CODEC>::kBytes;
  const int64_t blocks_per_row = columns / BV;
  const int64_t i = blockIdx.y;
  if (i >= count) return;
  const long long row = (long long)indexes[i];
  if (row < 0 || row >= rows) {  // recorded, never trapped: the host reports it after the stream sync
    if (threadIdx.x == 0 && blockIdx.x == 0 && atomicCAS(&status->code, kStatusNone, kStatusIndexOutOfRange) == kStatusNone) {
      status->value = row;
      status->bound = rows;
    }
    return;
  }
  for (int64_t col = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; col < columns; col += (int64_t)gridDim.x * blockDim.x) {
    const uint8_t* block = packed + (row * blocks_per_row + col / BV) * BB;
    out[i * columns + col] = decode_elem<CODEC>(block, (int)(col % BV));
  }
}

struct EmbeddingLaunch {
  const void* indexes; int is_i64; int64_t count; const uint8_t* weight; int64_t rows, columns; float* out;
  DeviceStatus* status; cudaStream_t stream; cudaError_t err;
  template <int CODEC> void operator()() {
    if (count == 0) { err = cudaSuccess; return; }
    const int threads = 256;
    dim3 grid((unsigned)std::min<int64_t>((columns + threads - 1) / threads, 64), (unsigned)count);
    if (is_i64)
      qembedding_kernel<CODEC, long long><<<grid, threads, 0, stream>>>((const long long*)indexes, count, weight, rows, columns, out, status);
    else
      qembedding_kernel<CODEC, unsigned int><<<grid, threads, 0, stream>>>((const unsigned int*)indexes, count, weight, rows, columns, out, status);
    err = cudaGetLastError();
  }
};
cudaError_t launch_qembedding(int codec, const void* indexes, int index_is_i64, int64_t count, const uint8_t* weight,
                              int64_t rows, int64_t columns, float* out, DeviceStatus* status, cudaStream_t stream) {
  EmbeddingLaunch l{indexes, index_is_i64, count, weight, rows, columns, out, status, stream, cudaSuccess};
  if (!dispatch_codec(codec, l)) return cudaErrorInvalidValue;
  return l.err;
}

// ============================================================================================
// Quantisers (the reference has none). Four threads per 32-value block, eight consecutive values each.
//   Q4_0: the element of largest magnitude, signed, divided by -8 is the scale d (so the extreme
//         maps to code 0); stored as f16; code = clamp(floor(x * (1/d) + 8.5), 0, 15) using the
//         unrounded f32 d; ties between equal magnitudes keep the first element.
//   Q8_0: d = absmax / 127 stored as f16; code = clamp(round-half-away(x * (1/d)), -127, 127).
// HBM-bound on the f32 input once the integer conversions are gone: a code is the low byte of value + 2^23 added with
// rounding down. A CTA takes 128 blocks, two 32-byte loads per thread in flight; the packed blocks are put together in
// shared memory (18 and 34 bytes fit no vector store) and leave as one contiguous 16-byte-wide copy. A warp per block with
// byte stores took 247 us (Q4_0) and 167 us (Q8_0) on [14336 x 4096] (235 MB in); this takes 49 and 51 us, 394 and 424 us on
// [128256 x 4096]. With two 16-byte loads per thread, which ask for every sector twice: 51 and 53, 435 and 451 us; they stay
// for inputs on a 16-byte boundary only.
// ============================================================================================
constexpr int kQuantThreads = 256;
constexpr int kQuantPasses = 2;
constexpr int kQuantBlocks = kQuantPasses * kQuantThreads / 4;  // per CTA

// floor of a value in [0, 2^22) in the low bits.
__device__ __forceinline__ uint32_t floor_bits(float v) { return __float_as_uint(__fadd_rd(v, 8388608.0f)); }
// The low bytes of four words.
__device__ __forceinline__ uint32_t low_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// Eight consecutive values from a 32-byte boundary in one request, read once.
__device__ __forceinline__ void load_eight(const float* src, float (&v)[8]) {
  asm volatile("ld.global.cs.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(src));
}

template <int CODEC>
__global__ void __launch_bounds__(kQuantThreads) quantize_kernel(const float* __restrict__ x, int64_t total_blocks, uint8_t* __restrict__ out) {
  constexpr int BB = CodecTraits<CODEC>::kBytes;
  __shared__ __align__(16) unsigned short stage[kQuantBlocks * BB / 2];
  const int64_t first = blockIdx.x * (int64_t)kQuantBlocks;
  const int blocks = (int)min((int64_t)kQuantBlocks, total_blocks - first);
  const int part = threadIdx.x & 3;
  const bool wide_in = (reinterpret_cast<uintptr_t>(x) & 15) == 0, widest_in = (reinterpret_cast<uintptr_t>(x) & 31) == 0;
  float v[kQuantPasses][8];
#pragma unroll
  for (int p = 0; p < kQuantPasses; ++p) {
    const int block = p * (kQuantThreads / 4) + (threadIdx.x >> 2);
    const float* src = x + (first + block) * 32 + part * 8;
    if (widest_in && block < blocks) {
      load_eight(src, v[p]);
      continue;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (block < blocks) q = wide_in ? __ldcs(reinterpret_cast<const float4*>(src) + h) : make_float4(src[4 * h], src[4 * h + 1], src[4 * h + 2], src[4 * h + 3]);
      v[p][4 * h] = q.x; v[p][4 * h + 1] = q.y; v[p][4 * h + 2] = q.z; v[p][4 * h + 3] = q.w;
    }
  }
#pragma unroll
  for (int p = 0; p < kQuantPasses; ++p) {
    const int block = p * (kQuantThreads / 4) + (threadIdx.x >> 2);
    // the block's value of largest magnitude, for Q8_0 its magnitude; a NaN is never taken
    float extreme = 0.0f;
    if (CODEC == kQ8_0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) extreme = fmaxf(extreme, fabsf(v[p][i]));
#pragma unroll
      for (int off = 1; off < 4; off <<= 1) extreme = fmaxf(extreme, __shfl_xor_sync(0xffffffffu, extreme, off));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (fabsf(v[p][i]) > fabsf(extreme)) extreme = v[p][i];
#pragma unroll
      for (int off = 1; off < 4; off <<= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, extreme, off);
        // the earlier element wins ties: it sits in the lower lane
        if (fabsf(o) > fabsf(extreme) || (fabsf(o) == fabsf(extreme) && (part & off))) extreme = o;
      }
    }
    uint32_t code[8], word[2];
    const float d = CODEC == kQ4_0 ? __fmul_rn(extreme, -0.125f)  // exact
                                   : __fdiv_rn(extreme, 127.0f);
    const float inv = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float scaled = __fmul_rn(v[p][i], inv);
      if (CODEC == kQ4_0) {
        code[i] = floor_bits(fminf(fmaxf(__fadd_rn(scaled, 8.5f), 0.0f), 15.5f));
      } else {  // half away from zero: floor(|x| + 1/2), the sum rounded down so that it cannot reach the next integer
        const uint32_t magnitude = floor_bits(__fadd_rd(fminf(fmaxf(fabsf(scaled), 0.0f), 127.0f), 0.5f));
        code[i] = scaled < 0.0f ? 0u - magnitude : magnitude;
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      word[h] = low_bytes(code[4 * h], code[4 * h + 1], code[4 * h + 2], code[4 * h + 3]);
      if (CODEC == kQ4_0) word[h] |= __shfl_down_sync(0xffffffffu, word[h], 2) << 4;  // values 16 on are the high nibbles
    }
    unsigned short* dst = stage + block * (BB / 2);
    if (part == 0) dst[0] = __half_as_ushort(__float2half_rn(d));
    if (CODEC == kQ8_0 || part < 2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        dst[1 + 4 * part + 2 * h] = (unsigned short)word[h];
        dst[2 + 4 * part + 2 * h] = (unsigned short)(word[h] >> 16);
      }
    }
  }
  __syncthreads();
  uint8_t* dst = out + first * BB;
  const int bytes = blocks * BB;
  const int wide = (reinterpret_cast<uintptr_t>(dst) & 15) == 0 ? bytes / 16 : 0;
  for (int i = threadIdx.x; i < wide; i += kQuantThreads) __stcs(reinterpret_cast<uint4*>(dst) + i, reinterpret_cast<const uint4*>(stage)[i]);
  for (int i = wide * 8 + threadIdx.x; i < bytes / 2; i += kQuantThreads) reinterpret_cast<unsigned short*>(dst)[i] = stage[i];
}

cudaError_t launch_quantize(int codec, const float* x, int64_t rows, int64_t columns, uint8_t* packed,
                            cudaStream_t stream) {
  const int64_t blocks = rows * (columns / 32);
  if (blocks == 0) return cudaSuccess;
  const unsigned grid = (unsigned)((blocks + kQuantBlocks - 1) / kQuantBlocks);
  if (codec == kQ4_0) quantize_kernel<kQ4_0><<<grid, kQuantThreads, 0, stream>>>(x, blocks, packed);
  else if (codec == kQ8_0) quantize_kernel<kQ8_0><<<grid, kQuantThreads, 0, stream>>>(x, blocks, packed);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

// ============================================================================================
// Generic linear on the raw GGUF layout (every codec). A warp walks RG rows, 1024 columns at a time: four windows of 256,
// eight threads to a window (Runs in codecs.cuh: header decoded once per 32 values, payload in 16-byte loads). A 16-byte
// activation load from shared memory, distinct in every thread, serves RG rows' packed f32 FMAs. Weights are decoded to
// f32 with at most one rounding less than the reference (scale * code + offset is one FMA), products and sums are f32.
// The activations are staged in the order the threads ask for them (the run layout is the codec's), once per CTA when
// they fit in kRawStageBytes, else in chunks of columns.
//
// What bounds it: latency. On Q4_K [14336 x 4096] with 5 vectors (the form for 6) 18.8 million warp instructions are issued, 10 per
// weight of a warp, which is 36 % of the schedulers' slots: 128 registers and the staged activations leave four warps to a scheduler, of
// which 3.2 are there on average (3584 row groups are 12.1 per CTA for eight warps, so that half of them idle in the second
// round), and the wait for a window's payload, requested when it is used, is the largest of their stalls (31 %). Of the issued
// ones each vector takes half an FMA per weight and 1 / (4 RG) of a shared-memory load (four cycles of the SM's one load path: RG = 4
// keeps that below the FMAs). Two CTAs per SM share the rows evenly. One warp per row that decoded value by value took 204 us on Q4_K
// [14336 x 4096] with 5 vectors (5 us of HBM); this takes 42 us, 20 with one vector.
// ============================================================================================
constexpr int kRawWarps = 8;
constexpr int kRawStageBytes = 96 * 1024;  // two CTAs per SM

__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

template <int CODEC, int VC, int RG, bool WIDE>
__global__ void __launch_bounds__(kRawWarps * 32, 2) qlinear_raw_kernel(const float* __restrict__ x, int vectors, int64_t columns,
                                                                        const uint8_t* __restrict__ weight, int64_t rows,
                                                                        const float* __restrict__ bias, float* __restrict__ out,
                                                                        int64_t out_stride, int chunk_windows) {
  extern __shared__ __align__(16) float4 staged[];  // [four windows][vector][8 quads][4 windows x 8 threads]
  constexpr int kValues = CodecTraits<CODEC>::kValues, kBytes = CodecTraits<CODEC>::kBytes;
  constexpr int kWindowBytes = 256 / kValues * kBytes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, s = lane & 7;
  const int v0 = blockIdx.y * VC;
  const int64_t row_bytes = columns / kValues * kBytes;
  const int windows = (int)((columns + 255) / 256);
  const bool wide_x = ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(columns * sizeof(float))) & 15) == 0;
  const int64_t groups = (rows + RG - 1) / RG;
  const int64_t g0 = groups * blockIdx.x / gridDim.x, g1 = groups * (blockIdx.x + 1) / gridDim.x;

  auto stage = [&](int w0, int here) {
    const int items = (here + 3) / 4 * VC * 256;
    for (int i = threadIdx.x; i < items; i += kRawWarps * 32) {
      const int t = i & 31, q = (i >> 5) & 7, v = (i >> 8) % VC, w = (i >> 8) / VC * 4 + (t >> 3);
      const int64_t c = (int64_t)(w0 + w) * 256 + run_column<CODEC>(t & 7, q >> 2) + 4 * (q & 3);
      float4 value = make_float4(0.f, 0.f, 0.f, 0.f);
      if (v0 + v < vectors && c < columns) {  // columns are whole blocks of 32: a quad is inside or outside as a whole
        const float* src = x + (int64_t)(v0 + v) * columns + c;
        value = wide_x ? *reinterpret_cast<const float4*>(src) : make_float4(src[0], src[1], src[2], src[3]);
      }
      staged[i] = value;
    }
  };
  const bool once = chunk_windows >= windows;
  if (once) {
    stage(0, windows);
    __syncthreads();
  }
  for (int64_t gb = g0; gb < g1; gb += kRawWarps) {
    const int64_t row0 = (gb + warp) * RG;
    const bool mine = gb + warp < g1;
    unsigned long long acc[RG][VC];
#pragma unroll
    for (int g = 0; g < RG; ++g)
#pragma unroll
      for (int v = 0; v < VC; ++v) acc[g][v] = 0ull;
    for (int w0 = 0; w0 < windows; w0 += chunk_windows) {
      const int here = min(chunk_windows, windows - w0);
      if (!once) {
        __syncthreads();
        stage(w0, here);
        __syncthreads();
      }
      if (!mine) continue;
      for (int w = 0; w < here; w += 4) {
        const int64_t window = w0 + w + (lane >> 3);
        if (w + (lane >> 3) >= here || (kValues == 32 && window * 256 + s * 32 >= columns)) continue;
        Runs runs[RG];
#pragma unroll
        for (int g = 0; g < RG; ++g) runs[g] = load_runs<CODEC, WIDE>(weight + min(row0 + g, rows - 1) * row_bytes + window * kWindowBytes, s);
        const ulonglong2* xs = reinterpret_cast<const ulonglong2*>(staged + (size_t)(w >> 2) * VC * 256 + lane);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          unsigned long long lo[RG], hi[RG];  // four decoded weights per row
#pragma unroll
          for (int g = 0; g < RG; ++g) {
            const int r = q >> 2;
            const uint32_t word = runs[g].code[r][q & 3];
            const unsigned long long sc = pack_f32x2(runs[g].scale[r], runs[g].scale[r]), of = pack_f32x2(runs[g].offset[r], runs[g].offset[r]);
            lo[g] = fma_f32x2(sc, pack_f32x2(run_code<CODEC>(word, 0), run_code<CODEC>(word, 1)), of);
            hi[g] = fma_f32x2(sc, pack_f32x2(run_code<CODEC>(word, 2), run_code<CODEC>(word, 3)), of);
          }
#pragma unroll
          for (int v = 0; v < VC; ++v) {
            const ulonglong2 xv = xs[(v * 8 + q) * 32];
#pragma unroll
            for (int g = 0; g < RG; ++g) acc[g][v] = fma_f32x2(hi[g], xv.y, fma_f32x2(lo[g], xv.x, acc[g][v]));
          }
        }
      }
    }
    if (!mine) continue;
#pragma unroll
    for (int g = 0; g < RG; ++g)
#pragma unroll
      for (int v = 0; v < VC; ++v) {
        float t = __uint_as_float((uint32_t)acc[g][v]) + __uint_as_float((uint32_t)(acc[g][v] >> 32));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
        if (lane == (g * VC + v) % 32 && row0 + g < rows && v0 + v < vectors) out[(int64_t)(v0 + v) * out_stride + row0 + g] = t + (bias ? bias[row0 + g] : 0.0f);
      }
  }
}

template <int CODEC, int VC, int RG>
cudaError_t launch_qlinear_raw(const float* x, int64_t vectors, int64_t columns, const uint8_t* weight, int64_t rows, const float* bias,
                               float* out, int64_t out_stride, int sm_count, cudaStream_t stream) {
  const int windows = (int)((columns + 255) / 256);
  const int chunk = std::min((windows + 3) / 4 * 4, kRawStageBytes / (VC * 4096) * 4);
  const bool wide = kWideBlocks<CODEC> && (reinterpret_cast<uintptr_t>(weight) & 15) == 0;
  auto kernel = wide ? qlinear_raw_kernel<CODEC, VC, RG, kWideBlocks<CODEC>> : qlinear_raw_kernel<CODEC, VC, RG, false>;
  const cudaError_t attr = opt_in_shared_memory(kernel, kRawStageBytes);
  if (attr != cudaSuccess) return attr;
  const int64_t groups = (rows + RG - 1) / RG;
  const unsigned grid = (unsigned)std::min<int64_t>((groups + kRawWarps - 1) / kRawWarps, 2 * sm_count);
  kernel<<<dim3(grid, (unsigned)((vectors + VC - 1) / VC)), kRawWarps * 32, (size_t)chunk * VC * 1024, stream>>>(x, (int)vectors, columns, weight, rows, bias,
                                                                                                                 out, out_stride, chunk);
  return cudaGetLastError();
}
// Rows of a warp: four, unless that leaves warps without any (below two rows for each of an SM's 16 warps).
template <int CODEC, int VC>
cudaError_t launch_qlinear_raw(const float* x, int64_t vectors, int64_t columns, const uint8_t* weight, int64_t rows, const float* bias,
                               float* out, int64_t out_stride, int sm_count, cudaStream_t stream) {
  if (rows > 32 * (int64_t)sm_count) return launch_qlinear_raw<CODEC, VC, 4>(x, vectors, columns, weight, rows, bias, out, out_stride, sm_count, stream);
  return launch_qlinear_raw<CODEC, VC, 1>(x, vectors, columns, weight, rows, bias, out, out_stride, sm_count, stream);
}

struct GenericLaunch {
  const float* x; int64_t vectors, columns; const uint8_t* weight; int64_t rows; const float* bias; float* out; int64_t out_stride;
  int sm_count; cudaStream_t stream; cudaError_t err; int launches;
  template <int CODEC> void operator()() {
    err = cudaSuccess;
    if (rows == 0 || vectors == 0) return;
    ++launches;
    // a pass over the weights serves up to 8 vectors; passes of one launch share their rows' bytes in L2
    if (vectors <= 1) err = launch_qlinear_raw<CODEC, 1>(x, vectors, columns, weight, rows, bias, out, out_stride, sm_count, stream);
    else if (vectors <= 2) err = launch_qlinear_raw<CODEC, 2>(x, vectors, columns, weight, rows, bias, out, out_stride, sm_count, stream);
    else if (vectors <= 4) err = launch_qlinear_raw<CODEC, 4>(x, vectors, columns, weight, rows, bias, out, out_stride, sm_count, stream);
    else if (vectors <= 6) err = launch_qlinear_raw<CODEC, 6>(x, vectors, columns, weight, rows, bias, out, out_stride, sm_count, stream);
    else err = launch_qlinear_raw<CODEC, 8>(x, vectors, columns, weight, rows, bias, out, out_stride, sm_count, stream);
  }
};
cudaError_t launch_qlinear_generic(int codec, const float* x, int64_t vectors, int64_t columns, const uint8_t* weight,
                                   int64_t rows, const float* bias, float* out, int sm_count, cudaStream_t stream, int* launches,
                                   int64_t out_stride) {
  GenericLaunch l{x, vectors, columns, weight, rows, bias, out, out_stride ? out_stride : rows, sm_count, stream, cudaSuccess, 0};
  if (!dispatch_codec(codec, l)) return cudaErrorInvalidValue;
  if (launches) *launches += l.launches;
  return l.err;
}

// ============================================================================================
// Tiled (128-row) weights: activations to f16, split-K sum, dispatch.
// ============================================================================================

// f32 [vectors, K] -> the hand-off layout [chunk of nv vectors][K/8][nv][8] f16, absent vectors zero. Cells are counted in 32
// bits: 2^32 of them would be 137 GB of input.
__global__ void hand_off_convert_kernel(const float* x, int vectors, int K, int nv_shift, int chunks, __half* xh) {
  chain_release();
  chain_wait();
  const unsigned k8 = K / 8, total = (chunks * k8) << nv_shift;
  for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const unsigned column = idx >> nv_shift, chunk = chunks > 1 ? column / k8 : 0u, kg = column - chunk * k8;
    const int v = (int)((chunk << nv_shift) + (idx & ((1u << nv_shift) - 1)));
    uint2 lo = make_uint2(0u, 0u), hi = lo;
    if (v < vectors) {
      lo = pack4(*reinterpret_cast<const float4*>(x + (size_t)v * K + kg * 8));
      hi = pack4(*reinterpret_cast<const float4*>(x + (size_t)v * K + kg * 8 + 4));
    }
    reinterpret_cast<uint4*>(xh)[idx] = make_uint4(lo.x, lo.y, hi.x, hi.y);
  }
}
cudaError_t launch_hand_off_convert(const float* x, int64_t vectors, int K, int nv, __half* xh, int sm_count, cudaStream_t stream) {
  int shift = 0;
  while (1 << shift < nv) ++shift;
  const int64_t chunks = (vectors + nv - 1) / nv, total = chunks * (K / 8) * nv;
  return launch_chained(hand_off_convert_kernel, dim3((unsigned)std::min<int64_t>((total + 255) / 256, 8 * sm_count)), dim3(256), 0, stream, x, (int)vectors, K,
                        shift, (int)chunks, xh);
}

// Sums the split-K partials [chunk of vpad vectors][split][vpad][rows_padded] in split order and applies bias / epilogue.
// `residual` and `out` may be the same buffer (the decoder adds projections onto its hidden state in place), so
// neither carries a no-alias promise.
__global__ void qlinear_reduce_kernel(const float* scratch, int splits, int vpad, int vectors, int rows,
                                      int rows_padded, const float* bias, const float* residual,
                                      int epilogue, float* out, __half* out_xh, int xh_nv) {
  chain_release();  // the next kernel of the step may be scheduled; it waits for this one before touching memory
  chain_wait();
  const int out_cols = epilogue == ETC_EPILOGUE_SWIGLU ? rows / 2 : rows;
  const int64_t total = (int64_t)vectors * out_cols;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int v = (int)(idx / out_cols), c = (int)(idx - (int64_t)v * out_cols);
    if (epilogue == ETC_EPILOGUE_SWIGLU) {
      const int r_gate = (c >> 3) * 16 + (c & 7), r_up = r_gate + 8;
      float gsum = 0.f, usum = 0.f;
      for (int s = 0; s < splits; ++s) {
        const float* p = scratch + ((size_t)(v / vpad * splits + s) * vpad + v % vpad) * rows_padded;
        gsum += p[r_gate];
        usum += p[r_up];
      }
      if (bias) { gsum += bias[r_gate]; usum += bias[r_up]; }
      const float act = silu_tanh(gsum) * usum;
      if (out) out[idx] = act;
      if (out_xh) out_xh[hand_off_cell(c >> 3, v, xh_nv, out_cols / 8) + (c & 7)] = half_sat(act);
    } else {
      float sum = 0.f;
      for (int s = 0; s < splits; ++s) sum += scratch[((size_t)(v / vpad * splits + s) * vpad + v % vpad) * rows_padded + c];
      if (bias) sum += bias[c];
      const float val = epilogue == ETC_EPILOGUE_RESIDUAL ? residual[idx] + sum : sum;
      out[idx] = val;
    }
  }
}

cudaError_t launch_qlinear_reduce(const float* scratch, int splits, int vpad, int vectors, int rows, int rows_padded,
                                  const float* bias, const float* residual, int epilogue, float* out, __half* out_xh, int xh_nv,
                                  cudaStream_t stream) {
  const int out_cols = epilogue == ETC_EPILOGUE_SWIGLU ? rows / 2 : rows;
  const int64_t total = (int64_t)vectors * out_cols;
  if (total == 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 8);
  return launch_chained(qlinear_reduce_kernel, dim3(grid), dim3(256), 0, stream, scratch, splits, vpad, vectors, rows, rows_padded, bias, residual,
                        epilogue, out, out_xh, xh_nv);
}

// Scratch layout of the tcgen05 path: [xh8 activations, rounded to 256 B][split-K partials].
static size_t umma_xh_region(const UmmaPlan& p) { return (p.xh_bytes + 255) & ~(size_t)255; }

size_t tiled_scratch_bytes(const TiledWeight& w, int64_t vectors, int sm_count) {
  if (vectors <= stream_max_vectors()) return stream_scratch_bytes(w, vectors, sm_count);
  const UmmaPlan p = plan_umma(w, vectors, sm_count);
  return umma_xh_region(p) + p.scratch_bytes;
}

cudaError_t launch_qlinear_tiled(const TiledWeight& w, const float* x, int64_t vectors, const float* bias,
                                 const float* residual, int epilogue, float* out, void* scratch, DeviceStatus* status,
                                 int sm_count, cudaStream_t stream, int* launches, const __half* xh_ready, __half* out_xh, int xh_nv,
                                 DeferredSum* defer) {
  if (defer) *defer = DeferredSum();
  if (vectors <= stream_max_vectors())
    return launch_qlinear_stream(w, x, xh_ready, vectors, bias, residual, epilogue, out, out_xh, scratch, status, sm_count, stream, launches, xh_nv, defer);
  const size_t xh_region = umma_xh_region(plan_umma(w, vectors, sm_count));  // f16 activations of every chunk, then the partials
  return launch_qlinear_umma(w, x, xh_ready, vectors, bias, residual, epilogue, out, out_xh, reinterpret_cast<__half*>(scratch),
                             reinterpret_cast<float*>(reinterpret_cast<char*>(scratch) + xh_region), status, sm_count, stream, launches);
}

}  // namespace etc
