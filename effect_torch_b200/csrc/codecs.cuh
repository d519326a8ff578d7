// Device decoders for GGUF block codecs. decode_elem<CODEC>(block, i) returns logical element i
// of one packed block with exactly the f32 operations, in the order, of the reference's
// decode_q*_k routines (crates/runtime-cpu/src/quantized.rs:117-261), so dequantised values are
// bit-identical: every multiply/subtract uses the non-contracting __fmul_rn / __fsub_rn
// intrinsics (the reference never fuses them). Q4_0 and Q8_0 follow the published 32-value block
// format: f16 scale first, then 16 nibble bytes (low nibbles = values 0..15, high nibbles =
// values 16..31, value = scale * (code - 8)) resp. 32 int8 (value = scale * code).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace etc {

enum : int { kQ4_0 = 2, kQ8_0 = 8, kQ2_K = 10, kQ3_K = 11, kQ4_K = 12, kQ5_K = 13, kQ6_K = 14 };

template <int CODEC> struct CodecTraits;
template <> struct CodecTraits<kQ4_0> { static constexpr int kValues = 32, kBytes = 18; };
template <> struct CodecTraits<kQ8_0> { static constexpr int kValues = 32, kBytes = 34; };
template <> struct CodecTraits<kQ2_K> { static constexpr int kValues = 256, kBytes = 84; };
template <> struct CodecTraits<kQ3_K> { static constexpr int kValues = 256, kBytes = 110; };
template <> struct CodecTraits<kQ4_K> { static constexpr int kValues = 256, kBytes = 144; };
template <> struct CodecTraits<kQ5_K> { static constexpr int kValues = 256, kBytes = 176; };
template <> struct CodecTraits<kQ6_K> { static constexpr int kValues = 256, kBytes = 210; };

__device__ __forceinline__ float fp16_at(const uint8_t* block, int offset) {
  const unsigned short bits = (unsigned short)(block[offset] | (block[offset + 1] << 8));
  return __half2float(__ushort_as_half(bits));
}

// quantized.rs:77-86
__device__ __forceinline__ void scale_min_k4(int index, const uint8_t* scales, int& scale, int& minimum) {
  if (index < 4) {
    scale = scales[index] & 63;
    minimum = scales[index + 4] & 63;
  } else {
    scale = (scales[index + 4] & 0x0f) | ((scales[index - 4] >> 6) << 4);
    minimum = (scales[index + 4] >> 4) | ((scales[index] >> 6) << 4);
  }
}

template <int CODEC>
__device__ __forceinline__ float decode_elem(const uint8_t* b, int i);

template <>
__device__ __forceinline__ float decode_elem<kQ4_0>(const uint8_t* b, int i) {
  const float d = fp16_at(b, 0);
  const int code = i < 16 ? (b[2 + i] & 0x0f) : (b[2 + i - 16] >> 4);
  return __fmul_rn(d, (float)(code - 8));
}

template <>
__device__ __forceinline__ float decode_elem<kQ8_0>(const uint8_t* b, int i) {
  const float d = fp16_at(b, 0);
  return __fmul_rn(d, (float)(int)(signed char)b[2 + i]);
}

// quantized.rs:117-138 — group order: half {0,1} x shift {0,2,4,6} x q_offset {0,16}
template <>
__device__ __forceinline__ float decode_elem<kQ2_K>(const uint8_t* b, int i) {
  const int group = i >> 4, within = i & 15;
  const int half = group >> 3, shift = ((group & 7) >> 1) * 2, q_offset = (group & 1) * 16;
  const float d = fp16_at(b, 80), dmin = fp16_at(b, 82);
  const int sc = b[group];
  const float dl = __fmul_rn(d, (float)(sc & 0x0f));
  const float ml = __fmul_rn(dmin, (float)(sc >> 4));
  const int q = (b[16 + half * 32 + q_offset + within] >> shift) & 3;
  return __fsub_rn(__fmul_rn(dl, (float)q), ml);
}

// quantized.rs:142-176
template <>
__device__ __forceinline__ float decode_elem<kQ3_K>(const uint8_t* b, int i) {
  const int group = i >> 4, within = i & 15;
  const int half = group >> 3, lane = (group & 7) >> 1, q_offset = (group & 1) * 16;
  const uint8_t* hmask = b;
  const uint8_t* quants = b + 32;
  const uint8_t* packed = b + 96;
  const float d = fp16_at(b, 108);
  const int low = group < 8 ? (packed[group] & 0x0f) : (packed[group - 8] >> 4);
  const int high = (packed[8 + (group & 3)] >> (2 * (group >> 2))) & 3;
  const int scale = (low | (high << 4)) - 32;
  const float dl = __fmul_rn(d, (float)scale);
  const int low_q = (quants[half * 32 + q_offset + within] >> (lane * 2)) & 3;
  const int high_q = (hmask[q_offset + within] & (1 << (half * 4 + lane))) == 0 ? 4 : 0;
  return __fmul_rn(dl, (float)(low_q - high_q));
}

// quantized.rs:180-199
template <>
__device__ __forceinline__ float decode_elem<kQ4_K>(const uint8_t* b, int i) {
  const int group = i >> 5, within = i & 31;
  const int pair = group >> 1, side = group & 1;
  const float d = fp16_at(b, 0), dmin = fp16_at(b, 2);
  int sc, mn;
  scale_min_k4(group, b + 4, sc, mn);
  const float dl = __fmul_rn(d, (float)sc), ml = __fmul_rn(dmin, (float)mn);
  const int raw = b[16 + pair * 32 + within];
  const int code = side == 0 ? (raw & 0x0f) : (raw >> 4);
  return __fsub_rn(__fmul_rn(dl, (float)code), ml);
}

// quantized.rs:203-234
template <>
__device__ __forceinline__ float decode_elem<kQ5_K>(const uint8_t* b, int i) {
  const int group = i >> 5, within = i & 31;
  const int pair = group >> 1, side = group & 1;
  const float d = fp16_at(b, 0), dmin = fp16_at(b, 2);
  int sc, mn;
  scale_min_k4(group, b + 4, sc, mn);
  const float dl = __fmul_rn(d, (float)sc), ml = __fmul_rn(dmin, (float)mn);
  const int raw = b[48 + pair * 32 + within];
  const int low_q = side == 0 ? (raw & 0x0f) : (raw >> 4);
  const int code = low_q + ((b[16 + within] & (1 << (pair * 2 + side))) == 0 ? 0 : 16);
  return __fsub_rn(__fmul_rn(dl, (float)code), ml);
}

// quantized.rs:238-261 — out index = half*128 + quarter*32 + index
template <>
__device__ __forceinline__ float decode_elem<kQ6_K>(const uint8_t* b, int i) {
  const int half = i >> 7, quarter = (i & 127) >> 5, index = i & 31;
  const uint8_t* ql = b + half * 64;
  const uint8_t* qh = b + 128 + half * 32;
  const float d = fp16_at(b, 208);
  const int low = (quarter & 1) ? ql[index + 32] : ql[index];
  const int low4 = (quarter & 2) ? (low >> 4) : (low & 0x0f);
  const int code = (low4 | (((qh[index] >> (2 * quarter)) & 3) << 4)) - 32;
  const int scale = (int)(signed char)b[192 + half * 8 + (index >> 4) + quarter * 2];
  return __fmul_rn(__fmul_rn(d, (float)scale), (float)code);
}

// ---------------------------------------------------------------------------------------------
// Runs: how a thread takes 32 of the 256 values of a window (one K-quant block, or eight 32-value blocks in a row) at
// once. Thread s of 8 gets two runs of 16 consecutive values that share one scale each: value = scale * code + offset with
// `code` = the stored byte minus kBias. The bytes of a run are 16 contiguous payload bytes in every format (a nibble, a
// 2-bit field or the whole byte of each), so the payload is one 16-byte load, and the header is decoded once per 32
// values instead of once per value.
struct Runs {
  uint32_t code[2][4];  // 16 bytes each, in column order
  float scale[2], offset[2];
};
template <int CODEC> struct RunTraits;
template <> struct RunTraits<kQ4_0> { static constexpr int kBias = 8; static constexpr bool kOffset = false; };
template <> struct RunTraits<kQ8_0> { static constexpr int kBias = 128; static constexpr bool kOffset = false; };
template <> struct RunTraits<kQ2_K> { static constexpr int kBias = 0; static constexpr bool kOffset = true; };
template <> struct RunTraits<kQ3_K> { static constexpr int kBias = 4; static constexpr bool kOffset = false; };
template <> struct RunTraits<kQ4_K> { static constexpr int kBias = 0; static constexpr bool kOffset = true; };
template <> struct RunTraits<kQ5_K> { static constexpr int kBias = 0; static constexpr bool kOffset = true; };
template <> struct RunTraits<kQ6_K> { static constexpr int kBias = 32; static constexpr bool kOffset = false; };

// First column, inside the window, of run r of thread s.
template <int CODEC>
__host__ __device__ __forceinline__ int run_column(int s, int r) {
  if (CODEC == kQ4_0 || CODEC == kQ8_0) return 32 * s + 16 * r;
  if (CODEC == kQ4_K || CODEC == kQ5_K) return 64 * (s >> 1) + 16 * (s & 1) + 32 * r;
  if (CODEC == kQ6_K) return 128 * (s >> 2) + 16 * (s & 3) + 64 * r;
  return 128 * (s >> 2) + 64 * ((s >> 1) & 1) + 16 * (s & 1) + 32 * r;  // Q2_K, Q3_K
}

// 16 bytes from any address, in aligned 4-byte words that each hold at least one of them; WIDE: from a 16-byte aligned
// one. Free of branches, so that the loads of several rows are in flight together.
template <bool WIDE>
__device__ __forceinline__ uint4 load16(const uint8_t* p) {
  if (WIDE) return *reinterpret_cast<const uint4*>(p);
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(at & ~(uintptr_t)3);
  const unsigned shift = 8u * (unsigned)(at & 3);
  const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[shift ? 4 : 3];
  return make_uint4(__funnelshift_r(w0, w1, shift), __funnelshift_r(w1, w2, shift), __funnelshift_r(w2, w3, shift), __funnelshift_r(w3, w4, shift));
}
// Whether a codec's header and payload stay 16-byte aligned behind an aligned first block.
template <int CODEC>
constexpr bool kWideBlocks = CODEC == kQ4_K || CODEC == kQ5_K;

// Thread s's runs of the window at `b`.
// WIDE: kWideBlocks, and the tensor is 16-byte aligned.
template <int CODEC, bool WIDE>
__device__ __forceinline__ Runs load_runs(const uint8_t* b, int s) {
  Runs o;
  if (CODEC == kQ4_0 || CODEC == kQ8_0) {
    b += s * CodecTraits<CODEC>::kBytes;
    o.scale[0] = o.scale[1] = fp16_at(b, 0);
    o.offset[0] = o.offset[1] = 0.0f;
    const uint4 q = load16<WIDE>(b + 2);
    const uint4 h = CODEC == kQ8_0 ? load16<WIDE>(b + 18) : q;
    const uint32_t lo[4] = {q.x, q.y, q.z, q.w}, hi[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o.code[0][j] = CODEC == kQ8_0 ? lo[j] ^ 0x80808080u : lo[j] & 0x0f0f0f0fu;
      o.code[1][j] = CODEC == kQ8_0 ? hi[j] ^ 0x80808080u : (hi[j] >> 4) & 0x0f0f0f0fu;
    }
  } else if (CODEC == kQ4_K || CODEC == kQ5_K) {
    const uint4 header = load16<WIDE>(b);  // d, dmin, 12 bytes of 6-bit scales and minima
    const int g = s >> 1, shift = 16 * (g & 1);
    const uint32_t a = header.y >> shift, m = header.z >> shift, x = header.w >> shift;
    const uint32_t sc = g < 2 ? a & 0x3f3fu : (x & 0x0f0fu) | ((a >> 2) & 0x3030u);
    const uint32_t mn = g < 2 ? m & 0x3f3fu : ((x >> 4) & 0x0f0fu) | ((m >> 2) & 0x3030u);
    const float d = __half2float(__ushort_as_half((unsigned short)header.x)), dmin = __half2float(__ushort_as_half((unsigned short)(header.x >> 16)));
    o.scale[0] = __fmul_rn(d, (float)(sc & 0xffu));
    o.scale[1] = __fmul_rn(d, (float)((sc >> 8) & 0xffu));
    o.offset[0] = -__fmul_rn(dmin, (float)(mn & 0xffu));
    o.offset[1] = -__fmul_rn(dmin, (float)((mn >> 8) & 0xffu));
    const uint4 q = load16<WIDE>(b + (CODEC == kQ4_K ? 16 : 48) + 16 * s);
    const uint4 h = CODEC == kQ5_K ? load16<WIDE>(b + 16 + 16 * (s & 1)) : q;
    const uint32_t lo[4] = {q.x, q.y, q.z, q.w}, hb[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o.code[0][j] = lo[j] & 0x0f0f0f0fu;
      o.code[1][j] = (lo[j] >> 4) & 0x0f0f0f0fu;
      if (CODEC == kQ5_K) {
        const uint32_t bits = hb[j] >> (2 * g);
        o.code[0][j] |= (bits & 0x01010101u) << 4;
        o.code[1][j] |= (bits & 0x02020202u) << 3;
      }
    }
  } else if (CODEC == kQ6_K) {
    const int half = s >> 2, first = 16 * (s & 3);  // first: 0..63 inside the half's 64 low-nibble bytes
    const uint4 q = load16<WIDE>(b + 64 * half + first), h = load16<WIDE>(b + 128 + 32 * half + (first & 31));
    const uint32_t lo[4] = {q.x, q.y, q.z, q.w}, hb[4] = {h.x, h.y, h.z, h.w};
    const int quarter = first >> 5;  // of the low nibbles; the high nibbles are two quarters on
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t bits = hb[j] >> (2 * quarter);
      o.code[0][j] = (lo[j] & 0x0f0f0f0fu) | ((bits & 0x03030303u) << 4);
      o.code[1][j] = ((lo[j] >> 4) & 0x0f0f0f0fu) | (bits & 0x30303030u);
    }
    const float d = fp16_at(b, 208);
    const uint8_t* scales = b + 192 + 8 * half + ((first & 31) >> 4) + 2 * quarter;
    o.scale[0] = __fmul_rn(d, (float)(int)(signed char)scales[0]);
    o.scale[1] = __fmul_rn(d, (float)(int)(signed char)scales[4]);
    o.offset[0] = o.offset[1] = 0.0f;
  } else {  // Q2_K, Q3_K: 2-bit fields, four to a byte
    const int half = s >> 2, field = 2 * ((s >> 1) & 1), within = s & 1;
    const uint4 q = load16<WIDE>(b + (CODEC == kQ2_K ? 16 : 32) + 32 * half + 16 * within);
    const uint4 h = CODEC == kQ3_K ? load16<WIDE>(b + 16 * within) : q;
    const uint32_t lo[4] = {q.x, q.y, q.z, q.w}, hb[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o.code[0][j] = (lo[j] >> (2 * field)) & 0x03030303u;
      o.code[1][j] = (lo[j] >> (2 * field + 2)) & 0x03030303u;
      if (CODEC == kQ3_K) {  // the high bit, set, stands for "no 4 to subtract"
        const uint32_t bits = hb[j] >> (4 * half + field);
        o.code[0][j] |= (bits & 0x01010101u) << 2;
        o.code[1][j] |= (bits & 0x02020202u) << 1;
      }
    }
    const int group = 8 * half + 2 * field + within;  // of 16 values; the second run's is two on
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int g = group + 2 * r;
      if (CODEC == kQ2_K) {
        const int sc = b[g];
        o.scale[r] = __fmul_rn(fp16_at(b, 80), (float)(sc & 0x0f));
        o.offset[r] = -__fmul_rn(fp16_at(b, 82), (float)(sc >> 4));
      } else {
        const uint8_t* packed = b + 96;
        const int low = g < 8 ? (packed[g] & 0x0f) : (packed[g - 8] >> 4);
        const int high = (packed[8 + (g & 3)] >> (2 * (g >> 2))) & 3;
        o.scale[r] = __fmul_rn(fp16_at(b, 108), (float)((low | (high << 4)) - 32));
        o.offset[r] = 0.0f;
      }
    }
  }
  return o;
}

// Byte j of a run's word as the f32 integer code: the byte lands in the mantissa of 2^23, which is subtracted again.
template <int CODEC>
__device__ __forceinline__ float run_code(uint32_t word, int j) {
  return __fadd_rn(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7440 + j)), -(8388608.0f + (float)RunTraits<CODEC>::kBias));
}
// The decoded value, with the reference's roundings.
template <int CODEC>
__device__ __forceinline__ float run_value(const Runs& o, int r, int i) {
  const float v = __fmul_rn(o.scale[r], run_code<CODEC>(o.code[r][i >> 2], i & 3));
  return RunTraits<CODEC>::kOffset ? __fadd_rn(v, o.offset[r]) : v;
}

// Runtime dispatch helper: calls f.template operator()<CODEC>() for a codec id; returns false
// for an unknown id.
template <typename F>
inline bool dispatch_codec(int codec, F&& f) {
  switch (codec) {
    case kQ4_0: f.template operator()<kQ4_0>(); return true;
    case kQ8_0: f.template operator()<kQ8_0>(); return true;
    case kQ2_K: f.template operator()<kQ2_K>(); return true;
    case kQ3_K: f.template operator()<kQ3_K>(); return true;
    case kQ4_K: f.template operator()<kQ4_K>(); return true;
    case kQ5_K: f.template operator()<kQ5_K>(); return true;
    case kQ6_K: f.template operator()<kQ6_K>(); return true;
    default: return false;
  }
}

}  // namespace etc
