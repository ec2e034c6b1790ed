// pm_mma.cuh -- exact products of residues by byte limbs on the int8 tensor
// cores, and Montgomery products, shared by the PM-basis kernels (pmleaf.cu,
// pmproduct.cu).
#pragma once
#include "rr_device.cuh"

namespace rr {

// D = A B (no accumulator to clear first)
__device__ __forceinline__ void mma_u8_first(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

// Montgomery products with the multiply-adds written in C: the compiler's wide
// multiply-adds issue at 3.6 cycles a warp and the whole redc2 returns after 29
// cycles, against 5.0 and 43 with mad.lo.cc / madc.hi chains (one warp per SM
// sub-partition; latency is what counts in these kernels).
__device__ __forceinline__ uint32_t redc_mul(uint32_t a, uint32_t b, const ModP& M) { return redc((uint64_t)a * b, M); }
__device__ __forceinline__ uint32_t redc2(uint32_t a, uint32_t b, uint32_t c, uint32_t d, const ModP& M) {
  return redc((uint64_t)c * d + (uint64_t)a * b, M);
}

// Word of (row, word) in a byte plane: the 8 rows x 4 words that a fragment
// load reads fall in 32 different banks.
template <int RL>
__device__ __forceinline__ int plane_word(int r, int w) {
  return RL == 1 ? r * 8 + (w ^ (((r >> 2) & 1) << 2)) : r * 16 + (w ^ (((r >> 1) & 3) << 2));
}

}  // namespace rr
