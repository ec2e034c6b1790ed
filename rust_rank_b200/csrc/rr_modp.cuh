// rr_modp.cuh -- exact arithmetic modulo a prime p < 2^31 on sm_100a.
//
// Values are kept as uint32 in [0, p).  Dot products and sparse row sums are
// accumulated lazily in 64 bits: a product of two residues is < p^2 < 2^62,
// and an accumulator is "folded" (hi * (2^32 mod p) + lo) after every
// `fold_every` products so that it never wraps.  The final residue comes from
// a Barrett reduction with mu = floor(2^64 / p) (Barrett, CRYPTO '86).
#pragma once
#include <cstdint>

namespace rr {

struct ModP {
  uint32_t p;      // the prime, p < 2^31
  uint32_t c32;    // 2^32 mod p
  uint64_t mu;     // floor(2^64 / p)
  uint32_t pinv;   // -p^{-1} mod 2^32 (Montgomery reduction with R = 2^32)
  uint32_t r1;     // R mod p
};

#ifdef __CUDACC__
// a * b + c exactly (mod 2^64).  Written in C: ptxas makes one wide multiply-add
// of it, which issues every 3.6 cycles per warp and SM sub-partition; the
// mad.lo.cc / madc.hi pair takes 5.0 (CUDA 12.9, B200).
__device__ __forceinline__ uint64_t mad_wide(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }

// Products of residues that fit a 64-bit accumulator between two folds, for every
// p < 2^31.  A folded accumulator is below 2^32 (c32 + 1).  For p = 2^31 - e > 2^32 / 3,
// c32 = 2e and 4 (p - 1)^2 = 2^64 - 2^32 (4e + 4) + (2e + 2)^2, together below 2^64
// because (2e + 2)^2 < 2^32 (2e + 3); for smaller p, 4 p^2 <= 4/9 2^64 and c32 < p.
constexpr int kFold = 4;

// Fold a 64-bit accumulator: result == x (mod p) and result < 2^32 * c32 + 2^32.
// Here the carry chain wins (mad_wide and fold of one accumulator 10.2 cycles
// against 11.8): the addend is half an accumulator, which the wide form has to
// be copied into a register pair for.
__device__ __forceinline__ uint64_t fold(uint64_t x, const ModP& M) {
  uint32_t lo = (uint32_t)x, hi = 0;
  asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.u32 %1, %2, %3, %1;"
      : "+r"(lo), "+r"(hi)
      : "r"((uint32_t)(x >> 32)), "r"(M.c32));
  return ((uint64_t)hi << 32) | lo;
}

// Exact x mod p for any 64-bit x.  q = floor(x*mu / 2^64) is at most 2 below
// floor(x/p), so r = x - q*p < 3p and two conditional subtractions finish.
__device__ __forceinline__ uint32_t reduce(uint64_t x, const ModP& M) {
  const uint64_t q = __umul64hi(x, M.mu);
  uint64_t r = x - q * (uint64_t)M.p;
  if (r >= M.p) r -= M.p;
  if (r >= M.p) r -= M.p;
  return (uint32_t)r;
}

// Montgomery reduction (Montgomery 1985), R = 2^32: for T < p * 2^32 returns
// T * R^{-1} mod p in [0, p).  m = T * (-p^{-1}) mod R makes T + m p divisible
// by R, and T + m p < 2 p R < 2^64.  A folded accumulator always satisfies
// the bound, since fold() < (2^32 - 1) * c32 + 2^32 <= (2^32 - 1) * p + 2^32 - 1.
__device__ __forceinline__ uint32_t redc(uint64_t T, const ModP& M) {
  const uint32_t m = (uint32_t)T * M.pinv;
  const uint64_t s = (uint64_t)m * M.p + T;
  const uint32_t t = (uint32_t)(s >> 32);
  return min(t, t - M.p);  // t < 2p
}

__device__ __forceinline__ uint32_t mulmod(uint32_t a, uint32_t b, const ModP& M) {
  return reduce((uint64_t)a * b, M);
}

__device__ __forceinline__ uint32_t addmod(uint32_t a, uint32_t b, uint32_t p) {
  const uint32_t s = a + b;  // a, b < 2^31 so no wrap
  return s >= p ? s - p : s;
}

__device__ __forceinline__ uint32_t submod(uint32_t a, uint32_t b, uint32_t p) {
  return a >= b ? a - b : a + p - b;
}
#endif  // __CUDACC__

}  // namespace rr
