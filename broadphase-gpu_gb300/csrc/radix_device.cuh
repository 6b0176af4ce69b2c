// radix_device.cuh - digits and in-warp ranking shared by the sorts.
#pragma once

#include "stq_device.cuh"

namespace stq {

constexpr int kRadixBins = 256;

// Digit of a key (digits are whole bytes).
__device__ __forceinline__ unsigned digit_of(uint32_t k, int shift) { return __byte_perm(k, 0, 0x4440 | (shift >> 3)); }
__device__ __forceinline__ unsigned digit_of(unsigned long long k, int shift) {
  return digit_of(shift >= 32 ? uint32_t(k >> 32) : uint32_t(k), shift & 31);
}

// Lanes of the warp whose digit is d: one ballot per bit, four instructions
// each. The ranking is what bounds a pass (the integer pipe is 70% busy), and
// __match_any_sync is slower: 92 M pairs take 4.68 ms with it, 3.51 with
// ballots as the compiler writes them, 3.16 with these.
__device__ __forceinline__ unsigned same_digit(unsigned d) {
  unsigned m = kFullMask;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    unsigned v, s;  // v: lanes whose bit is set; s: 0 if this lane's is, else all ones
    asm volatile(
        "{ .reg .pred p; .reg .b32 t; and.b32 t, %2, %3; setp.ne.u32 p, t, 0;\n"
        "vote.sync.ballot.b32 %0, p, 0xffffffff; selp.b32 %1, 0, 0xffffffff, p; }"
        : "=r"(v), "=r"(s)
        : "r"(d), "r"(1u << b));
    m &= v ^ s;
  }
  return m;
}

}  // namespace stq
