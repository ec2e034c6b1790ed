// pm_mma.cuh -- exact products of residues by byte limbs on the int8 tensor
// cores, and Montgomery products, shared by the PM-basis kernels (pmleaf.cu,
// pmproduct.cu).
#pragma once
#include "rr_modp.cuh"

namespace rr {

// D = A B (no accumulator to clear first)
__device__ __forceinline__ void mma_u8_first(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_u8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Montgomery products with the multiply-adds written in C: in the
// PM-basis kernels the compiler's wide multiply-adds issue at 3.6 cycles a warp and the whole
// redc2 returns after 29 cycles, against 5.0 and 43 with mad.lo.cc / madc.hi
// chains (one warp per SM sub-partition; latency is what counts here).
__device__ __forceinline__ uint32_t redc64(uint64_t T, const ModP& M) {  // T < p 2^32
  const uint32_t q = (uint32_t)T * M.pinv;
  const uint32_t t = (uint32_t)(((uint64_t)q * M.p + T) >> 32);
  return min(t, t - M.p);
}
__device__ __forceinline__ uint32_t redc_mul(uint32_t a, uint32_t b, const ModP& M) { return redc64((uint64_t)a * b, M); }
__device__ __forceinline__ uint32_t redc2(uint32_t a, uint32_t b, uint32_t c, uint32_t d, const ModP& M) {
  return redc64((uint64_t)c * d + (uint64_t)a * b, M);
}

// Word of (row, word) in a byte plane: the 8 rows x 4 words that a fragment
// load reads fall in 32 different banks.
template <int RL>
__device__ __forceinline__ int plane_word(int r, int w) {
  return RL == 1 ? r * 8 + (w ^ (((r >> 2) & 1) << 2)) : r * 16 + (w ^ (((r >> 1) & 3) << 2));
}
__device__ __forceinline__ void byte_transpose4(const uint32_t (&v)[4], uint32_t (&w)[4]) {
  // w[l] = bytes l of v[0..3]
  const uint32_t t0 = __byte_perm(v[0], v[1], 0x5140), t1 = __byte_perm(v[2], v[3], 0x5140);
  const uint32_t t2 = __byte_perm(v[0], v[1], 0x7362), t3 = __byte_perm(v[2], v[3], 0x7362);
  w[0] = __byte_perm(t0, t1, 0x5410);
  w[1] = __byte_perm(t0, t1, 0x7632);
  w[2] = __byte_perm(t2, t3, 0x5410);
  w[3] = __byte_perm(t2, t3, 0x7632);
}

}  // namespace rr
