// divmagic.h - signed 32-bit division and remainder by a divisor fixed per style, through a
// multiply-high with a precomputed magic number (Warren, "Hacker's Delight", section 10-1: signed
// division by constants). Exact for every int32 dividend, with C's truncating semantics, so it
// replaces `n % d` bit for bit while keeping the per-pixel remainder off the slow division path.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define BLGPU_HD __host__ __device__ __forceinline__
#else
#define BLGPU_HD inline
#endif

namespace blgpu {

struct DivMagic {
  int32_t m;       // magic multiplier
  int32_t s;       // post-shift; -1: the divisor is 1 (remainder 0)
};

// Magic number and shift for a divisor d >= 1 (Granlund and Montgomery, "Division by Invariant Integers
// using Multiplication", 1994, section 5): with l = ceil(log2 d), m = floor(2^(31 + l) / d) + 1 - 2^32 and
// shift l - 1, the quotient is n plus the high product, shifted, plus 1 for a negative n. One division and
// no search: one for the smallest shift, or for l, takes 30 steps for the 2^31 - 1 that stands for "no wrap".
inline DivMagic div_magic(int32_t d) {
  if (d == 1) return DivMagic{0, -1};
  const int32_t l = 32 - __builtin_clz(uint32_t(d - 1));
  return DivMagic{int32_t(uint32_t((uint64_t(1) << (31 + l)) / uint32_t(d) + 1u)), l - 1};
}

BLGPU_HD int32_t mulhi_s32(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return int32_t((int64_t(a) * int64_t(b)) >> 32);
#endif
}

// n % d (C semantics) for d >= 1 with dm = div_magic(d).
BLGPU_HD int32_t smod_magic(int32_t n, int32_t d, DivMagic dm) {
  if (dm.s < 0) return 0;
  int32_t q = mulhi_s32(dm.m, n);
  if (dm.m < 0) q += n;
  q >>= dm.s;
  q += int32_t(uint32_t(n) >> 31);
  return int32_t(uint32_t(n) - uint32_t(q) * uint32_t(d));
}

}  // namespace blgpu
