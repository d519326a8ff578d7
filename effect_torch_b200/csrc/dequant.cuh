// What the tcgen05 linears share: the expansion of packed weight blocks to f16 in registers, ring positions and warp-wide
// bounded waits.
#pragma once

#include "tc05.cuh"

namespace etc {
namespace tc05 {

// Bounded wait of a whole warp: one poll and a vote when the phase is over already.
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_try_wait(bar, parity)) || mbar_wait_warp(bar, parity, abort_flag);
}

// The position of a ring of N buffers: index and the parity of its current round.
template <int N>
struct Ring {
  int at = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next() {
    if (++at == N) { at = 0; parity ^= 1u; }
  }
  __device__ __forceinline__ void skip(int n) {  // n <= N
    at += n;
    if (at >= N) { at -= N; parity ^= 1u; }
  }
};

// Codes in the tiled layout stand where a masked word reads as f16: bits 0 to 10 of a half count in units of 2^-24 whether the
// half is subnormal or in the first normal binade, so a code at bit p is the f16 number code * 2^(p - 24). One FMA then scales
// it and subtracts the offset, with the one rounding that scaling the whole-number code has:
//     weight = code * 2^(p - 24) * (scale * 2^(24 - p)) - offset * scale,
// in which all products are exact while scale * 2^21 is a finite f16. Larger scales (2^-5 and more) take a second form with
// the same results. (Splicing codes into the mantissa of 1024, taking 1024 off again and scaling cost 8 FMAs for eight 4-bit
// codes where this costs 4; a dequant warp had 366 instructions per stage of 128 x 128 weights, now 255.)
__device__ __forceinline__ uint32_t mul_h2(uint32_t x, uint32_t y) {
  uint32_t d;
  asm("mul.f16x2 %0, %1, %2;" : "=r"(d) : "r"(x), "r"(y));
  return d;
}
__device__ __forceinline__ uint32_t fma_h2(uint32_t x, uint32_t y, uint32_t z) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(y), "r"(z));
  return d;
}

// Masks of the code pairs in a word and in the word rotated right by 8: 4-bit codes at bits 3 and 7 of a half, bytes at bit 3.
constexpr uint32_t kCodesLow = 0x00780078u, kCodesHigh = 0x07800780u, kBytes = 0x07F807F8u;
__device__ __forceinline__ uint32_t rotate8(uint32_t q) { return __funnelshift_r(q, q, 8); }

// Of a codec in the tiled layout: 4-bit codes or bytes, one f16 or two per block, the second a minimum or the second half's
// scale, and what is taken off a code.
template <int CODEC>
struct Coding {
  static constexpr bool kNibbles = CODEC == 2 || CODEC == 12, kPair = CODEC >= 12, kMinimum = CODEC == 12 || CODEC == 13;
  static constexpr int kOffset = kMinimum ? 0 : (kNibbles ? 8 : 128);
};

// The scales of a block at s, each twice in a register.
template <int CODEC>
__device__ __forceinline__ void load_scales(const unsigned char* s, uint32_t& scale, uint32_t& second) {
  const uint32_t raw = Coding<CODEC>::kPair ? *reinterpret_cast<const uint32_t*>(s) : (uint32_t)*reinterpret_cast<const unsigned short*>(s);
  scale = __byte_perm(raw, raw, 0x1010);
  second = Coding<CODEC>::kPair ? __byte_perm(raw, raw, 0x3232) : 0u;
}

// The magnitude of x or y, whichever is larger (the sign means nothing); a NaN gives way to the other.
__device__ __forceinline__ uint32_t larger_h2(uint32_t x, uint32_t y) {
  uint32_t d;
  asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(d) : "r"(x), "r"(y));
  return d;
}
// Whether every lane's scales of N blocks are below 2^-5 (or NaN, which both forms carry through).
template <int CODEC, int N>
__device__ __forceinline__ bool small_scales(const uint32_t (&scale)[N], const uint32_t (&second)[N]) {
  uint32_t most = scale[0];
#pragma unroll
  for (int b = 1; b < N; ++b) most = larger_h2(most, scale[b]);
  if (CODEC == 14)
#pragma unroll
    for (int b = 0; b < N; ++b) most = larger_h2(most, second[b]);
  return __all_sync(0xffffffffu, (most & 0x7fffu) < 0x2800u || (most & 0x7fffu) > 0x7c00u);
}

// What one word's codes need of their scale.
template <int CODEC, bool LARGE>
struct Factors {
  uint32_t scale, low, high, bias;
  __device__ __forceinline__ Factors(uint32_t s, uint32_t minimum) : scale(s) {
    if (LARGE) {
      bias = minimum ^ 0x80008000u;
    } else {
      const uint32_t part = mul_h2(s, 0x68006800u);                       // * 2^11
      low = mul_h2(part, 0x64006400u);                                    // * 2^21
      high = Coding<CODEC>::kNibbles ? mul_h2(part, 0x54005400u) : 0u;    // * 2^17
      bias = Coding<CODEC>::kMinimum ? minimum ^ 0x80008000u : mul_h2(s, Coding<CODEC>::kOffset == 8 ? 0xC800C800u : 0xD800D800u);
    }
  }
  // masked codes at bit 3 (HIGH: 7) of each half -> weights
  template <bool HIGH>
  __device__ __forceinline__ uint32_t weights(uint32_t codes) const {
    if (!LARGE) return fma_h2(codes, HIGH ? high : low, bias);
    // * 2^15 and * 2^6 (2^2): the whole-number code, less its offset
    constexpr int kOffset = Coding<CODEC>::kOffset;
    const uint32_t off = kOffset == 0 ? 0u : kOffset == 8 ? (HIGH ? 0xC000C000u : 0xB000B000u) : 0xC000C000u;  // -2, -1/8; -2
    const uint32_t whole = mul_h2(fma_h2(codes, 0x78007800u, off), HIGH ? 0x44004400u : 0x54005400u);
    return Coding<CODEC>::kMinimum ? fma_h2(whole, scale, bias) : mul_h2(whole, scale);
  }
};

// One 32-value block of one row in the tiled layout (packed words at q) -> 16 half2 in column order.
template <int CODEC, bool LARGE>
__device__ __forceinline__ void expand_block(const unsigned char* q, uint32_t scale, uint32_t second, uint32_t (&regs)[16]) {
  const uint4 a = *reinterpret_cast<const uint4*>(q);
  const uint32_t lo[4] = {a.x, a.y, a.z, a.w};
  const Factors<CODEC, LARGE> f(scale, second);
  if constexpr (Coding<CODEC>::kNibbles) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t r = rotate8(lo[j]);
      regs[4 * j] = f.template weights<false>(lo[j] & kCodesLow);
      regs[4 * j + 1] = f.template weights<false>(r & kCodesLow);
      regs[4 * j + 2] = f.template weights<true>(lo[j] & kCodesHigh);
      regs[4 * j + 3] = f.template weights<true>(r & kCodesHigh);
    }
  } else {
    const uint4 b = *reinterpret_cast<const uint4*>(q + 16);
    const uint32_t hi[4] = {b.x, b.y, b.z, b.w};
    const Factors<CODEC, LARGE> g(CODEC == 14 ? second : scale, second);  // the same as f but for two scales per block
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      regs[2 * j] = f.template weights<false>(lo[j] & kBytes);
      regs[2 * j + 1] = f.template weights<false>(rotate8(lo[j]) & kBytes);
      regs[8 + 2 * j] = g.template weights<false>(hi[j] & kBytes);
      regs[8 + 2 * j + 1] = g.template weights<false>(rotate8(hi[j]) & kBytes);
    }
  }
}

// One block of Q4_0 or Q8_0 -> 16 half2 of whole-number codes / 64, which the block's f32 scale makes up for. (Left at 2^-17
// the codes would be subnormal, and the tensor core aligns the products of subnormals by their exponent field: three bits of
// the sum lost.)
constexpr float kCodeUnits = 64.0f;
template <int CODEC>
__device__ __forceinline__ void expand_codes(const unsigned char* q, uint32_t (&regs)[16]) {
  static_assert(CODEC == 2 || CODEC == 8, "one scale per block");
  constexpr uint32_t kOff = CODEC == 2 ? 0xB000B000u : 0xC000C000u;  // -8 / 64, -128 / 64
  const uint4 a = *reinterpret_cast<const uint4*>(q);
  const uint32_t lo[4] = {a.x, a.y, a.z, a.w};
  if (CODEC == 2) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t r = rotate8(lo[j]);
      regs[4 * j] = fma_h2(lo[j] & kCodesLow, 0x78007800u, kOff);  // * 2^15
      regs[4 * j + 1] = fma_h2(r & kCodesLow, 0x78007800u, kOff);
      regs[4 * j + 2] = fma_h2(lo[j] & kCodesHigh, 0x68006800u, kOff);  // * 2^11
      regs[4 * j + 3] = fma_h2(r & kCodesHigh, 0x68006800u, kOff);
    }
  } else {
    const uint4 b = *reinterpret_cast<const uint4*>(q + 16);
    const uint32_t hi[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      regs[2 * j] = fma_h2(lo[j] & kBytes, 0x78007800u, kOff);
      regs[2 * j + 1] = fma_h2(rotate8(lo[j]) & kBytes, 0x78007800u, kOff);
      regs[8 + 2 * j] = fma_h2(hi[j] & kBytes, 0x78007800u, kOff);
      regs[8 + 2 * j + 1] = fma_h2(rotate8(hi[j]) & kBytes, 0x78007800u, kOff);
    }
  }
}

}  // namespace tc05
}  // namespace etc
