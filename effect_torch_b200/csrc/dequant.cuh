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

// Splice constants as launch arguments, so that the compiler keeps them in registers: a three-input logic operation or an
// f16x2 FMA has room for one immediate, and every second one costs an instruction (the ALU pipe, which does the splicing at
// half rate, was 59 % busy with them, 436 instructions per warp and stage of 128 x 128 weights).
struct Splice {
  uint32_t magic = 0x64006400u;      // half2(1024, 1024): a code spliced into the mantissa reads 1024 + code
  uint32_t mask_lo = 0x000F000Fu, mask_hi = 0x00F000F0u;
  uint32_t sixteenth = 0x2C002C00u;  // half2(1/16, 1/16)
  uint32_t bias_lo = 0xE408E408u, bias_hi = 0xD480D480u;      // half2(-1032), half2(-72): Q4_0 codes minus 8
  uint32_t bias_lo_k = 0xE400E400u, bias_hi_k = 0xD400D400u;  // half2(-1024), half2(-64): unsigned codes
  uint32_t bias_byte = 0xE480E480u;  // half2(-1152): bytes plus 128
  uint32_t fill = 0x64646464u, flip = 0x80808080u;
};
__device__ __forceinline__ uint32_t and_or(uint32_t x, uint32_t mask, uint32_t fill) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(x), "r"(mask), "r"(fill));  // (x & mask) | fill
  return d;
}
__device__ __forceinline__ uint32_t add_h2(uint32_t x, uint32_t y) {
  uint32_t d;
  asm("add.f16x2 %0, %1, %2;" : "=r"(d) : "r"(x), "r"(y));
  return d;
}
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
// One packed word of eight 4-bit codes, logical column j at bit {0,16,8,24,4,20,12,28}[j] -> four half2 in column order,
// scaled; OFFSET: plus `second`. RAW: the whole-number codes themselves.
template <bool OFFSET, bool RAW = false>
__device__ __forceinline__ void splice_nibbles(uint32_t q, uint32_t scale, uint32_t second, const Splice& k, uint32_t* out) {
  const uint32_t qs = q >> 8;
  const uint32_t lo = OFFSET ? k.bias_lo_k : k.bias_lo, hi = OFFSET ? k.bias_hi_k : k.bias_hi;
  const uint32_t c0 = add_h2(and_or(q, k.mask_lo, k.magic), lo), c1 = add_h2(and_or(qs, k.mask_lo, k.magic), lo);
  const uint32_t c2 = fma_h2(and_or(q, k.mask_hi, k.magic), k.sixteenth, hi), c3 = fma_h2(and_or(qs, k.mask_hi, k.magic), k.sixteenth, hi);
  if (RAW) { out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3; return; }
  out[0] = OFFSET ? fma_h2(c0, scale, second) : mul_h2(c0, scale);
  out[1] = OFFSET ? fma_h2(c1, scale, second) : mul_h2(c1, scale);
  out[2] = OFFSET ? fma_h2(c2, scale, second) : mul_h2(c2, scale);
  out[3] = OFFSET ? fma_h2(c3, scale, second) : mul_h2(c3, scale);
}
// One word of four int8 codes -> two half2.
template <bool OFFSET, bool RAW = false>
__device__ __forceinline__ void splice_bytes(uint32_t w, uint32_t scale, uint32_t second, const Splice& k, uint32_t* out) {
  const uint32_t x = w ^ k.flip;
  const uint32_t c0 = add_h2(__byte_perm(x, k.fill, 0x4140), k.bias_byte), c1 = add_h2(__byte_perm(x, k.fill, 0x4342), k.bias_byte);
  if (RAW) { out[0] = c0; out[1] = c1; return; }
  out[0] = OFFSET ? fma_h2(c0, scale, second) : mul_h2(c0, scale);
  out[1] = OFFSET ? fma_h2(c1, scale, second) : mul_h2(c1, scale);
}

// One 32-value block of one row of Q4_0 or Q8_0 in the tiled layout -> 16 half2 of whole-number codes.
template <int CODEC>
__device__ __forceinline__ void expand_codes(const unsigned char* q, const Splice& k, uint32_t (&regs)[16]) {
  static_assert(CODEC == 2 || CODEC == 8, "one scale per block");
  const uint4 a = *reinterpret_cast<const uint4*>(q);
  const uint32_t lo[4] = {a.x, a.y, a.z, a.w};
  if (CODEC == 2) {
#pragma unroll
    for (int j = 0; j < 4; ++j) splice_nibbles<false, true>(lo[j], 0u, 0u, k, regs + 4 * j);
  } else {
    const uint4 b = *reinterpret_cast<const uint4*>(q + 16);
    const uint32_t hi[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) splice_bytes<false, true>(lo[j], 0u, 0u, k, regs + 2 * j);
#pragma unroll
    for (int j = 0; j < 4; ++j) splice_bytes<false, true>(hi[j], 0u, 0u, k, regs + 8 + 2 * j);
  }
}

// One 32-value block of one row in the tiled layout: packed words at q, block scale(s) at s -> 16 half2, scaled.
template <int CODEC>
__device__ __forceinline__ void expand_block(const unsigned char* q, const unsigned char* s, const Splice& k, uint32_t (&regs)[16]) {
  constexpr bool kPair = CODEC >= 12, kOffset = CODEC == 12 || CODEC == 13;
  const uint32_t sraw = kPair ? *reinterpret_cast<const uint32_t*>(s) : (uint32_t)*reinterpret_cast<const unsigned short*>(s);
  const uint32_t scale = __byte_perm(sraw, sraw, 0x1010);
  // the block's minimum, negated, or the scale of its second half
  const uint32_t second = kPair ? __byte_perm(sraw, sraw, 0x3232) ^ (kOffset ? 0x80008000u : 0u) : 0u;
  const uint4 a = *reinterpret_cast<const uint4*>(q);
  const uint32_t lo[4] = {a.x, a.y, a.z, a.w};
  if (CODEC == 2 || CODEC == 12) {
#pragma unroll
    for (int j = 0; j < 4; ++j) splice_nibbles<kOffset>(lo[j], scale, second, k, regs + 4 * j);
  } else {
    const uint4 b = *reinterpret_cast<const uint4*>(q + 16);
    const uint32_t hi[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) splice_bytes<kOffset>(lo[j], scale, second, k, regs + 2 * j);
#pragma unroll
    for (int j = 0; j < 4; ++j) splice_bytes<kOffset>(hi[j], CODEC == 14 ? second : scale, second, k, regs + 8 + 2 * j);
  }
}

}  // namespace tc05
}  // namespace etc
