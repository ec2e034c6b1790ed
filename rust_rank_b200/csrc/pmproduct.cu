// pmproduct.cu -- short products of polynomial matrices on the int8 tensor
// cores: C[t] = sum_s A[s] B[t - s] directly, in one launch.
//
// Above its leaf blocks the PM-basis multiplies matrices of 2b x 2b polynomials
// with a few dozen coefficients many times.  Through transforms such a product
// is four launches of a few microseconds' latency each (two forward, pointwise,
// inverse); as a block product it is little work for the tensor cores.  With
// byte limbs A = sum_a 256^a A_a the products of a limb class a + b are summed
// over the inner dimension AND over s in int32 -- at most (h + 1) r 4 255^2 <
// 2^29.1 for the sizes taken (direct_product_max) -- so the limbs are joined
// once per coefficient of the result, not once per term.
//
// A CTA computes a 16 x 8 tile of TC coefficients: it lays out the byte planes
// of its 16 rows of A (all coefficients) and 8 columns of B (those it needs) in
// shared memory, then each warp sums the terms s = sp mod SS of one coefficient
// and the SS partial sums are added mod p.  Inner dimensions up to 16 take two
// limb pairs per k-step (10 products per term instead of 16).
//
// Measured (mean over the two products of a level, one generator; before: the
// four launches of the transform path at twice the present length, 50 us on the
// mean over all levels): r = 32, h = 32 and 64: 15 us; r = 16, h = 64 and 128:
// 15 us; r = 64, h = 16 and 32: 23 us.  The tensor pipe bounds it (17 terms of
// 16 products of 16 cycles for each of 4 warps of an SM sub-partition at h = 64),
// then the load of the planes.
#include <algorithm>

#include "pm_mma.cuh"
#include "pmproduct.h"

namespace rr {

namespace {

constexpr int kThreads = 512;
constexpr int TC = 4;                       // coefficients per CTA
constexpr int SS = kThreads / 32 / TC;      // warps that share a coefficient
constexpr size_t kSmemLimit = 227 * 1024 - 1024;

// CFG 0: inner dimension <= 16, 1: <= 32, 2: <= 64.  Words of a plane row, of
// one coefficient of A (16 rows) and of B (8 columns); the odd strides put the
// same word of neighbouring coefficients in different banks.
template <int CFG>
struct ProductShape {
  static constexpr int KW = CFG == 0 ? 4 : CFG == 1 ? 8 : 16;
  static constexpr int AW = 64 * KW + 1, BW = 32 * KW + 1;
  static __device__ __forceinline__ int word(int r, int w) {
    if constexpr (CFG == 0) return r * 4 + w;
    else return plane_word<CFG == 0 ? 1 : CFG>(r, w);
  }
};
constexpr int kRedWords = SS * TC * 128;

template <int CFG>
constexpr size_t product_smem(int h) {
  return 4 * ((size_t)(h + 1) * ProductShape<CFG>::AW + (size_t)(h + TC) * ProductShape<CFG>::BW + kRedWords);
}
static_assert(product_smem<0>(128) <= kSmemLimit && product_smem<1>(64) <= kSmemLimit &&
                  product_smem<2>(32) <= kSmemLimit,
              "shared memory");

// The byte planes of `rows` x r entries (row `row`, inner index q at src + row *
// row_stride + q * in_stride) of `count` coefficients from t0 on.
template <int CFG>
__device__ __forceinline__ void load_planes(uint32_t* dst, int stride, const uint32_t* src, int rows_used, int rows,
                                            int64_t row_stride, int r, int64_t in_stride, int t0, int count) {
  using S = ProductShape<CFG>;
  // an item is one word of a plane row (four inner indices) of one coefficient;
  // four items of a thread are in flight
  const int total = rows * S::KW * count;
  const uint32_t inv = count > 1 ? 0xffffffffu / (uint32_t)count + 1 : 0u;  // exact: items * count < 2^32
  for (int e0 = threadIdx.x; e0 < total; e0 += 4 * kThreads) {
    uint32_t v[4][4];
    int q[4], c[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * kThreads;
      q[u] = count > 1 ? (int)__umulhi((uint32_t)e, inv) : e;
      c[u] = e - q[u] * count;
      const int row = q[u] / S::KW, w = q[u] % S::KW;
      const bool on = e < total && row < rows_used;
      const uint32_t* p = src + row * row_stride + (int64_t)4 * w * in_stride + t0 + c[u];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[u][j] = on && 4 * w + j < r ? p[j * in_stride] : 0u;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (e0 + u * kThreads >= total) break;
      uint32_t b[4];
      byte_transpose4(v[u], b);
      uint32_t* d = dst + (size_t)c[u] * stride + S::word(q[u] / S::KW, q[u] % S::KW);
#pragma unroll
      for (int l = 0; l < 4; ++l) d[l * rows * S::KW] = b[l];
    }
  }
}

template <int CFG>
__global__ void __launch_bounds__(kThreads, 1) direct_product_kernel(DirectProduct P) {
  using S = ProductShape<CFG>;
  extern __shared__ __align__(16) uint32_t pp_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int jtiles = (P.k + 7) / 8;
  const int strip = blockIdx.y / jtiles, jt = blockIdx.y % jtiles;
  const int t0 = P.lo + blockIdx.x * TC;                       // first coefficient of the CTA
  const int t_end = min(t0 + TC, P.lo + P.cnt);
  const uint32_t* A = P.A + blockIdx.z * P.a_bs + (int64_t)strip * 16 * P.a_rs;
  const uint32_t* Bm = P.B + blockIdx.z * P.b_bs + (int64_t)jt * 8 * P.b_cs;
  const ModP M = P.M;
  // terms of any of the CTA's coefficients: s in [s0, s1], u = t - s in [u0, u1]
  const int s0 = max(0, t0 - (P.lb - 1)), s1 = min(P.la - 1, t_end - 1);
  const int u0 = max(0, t0 - s1), u1 = min(P.lb - 1, t_end - 1 - s0);
  uint32_t* const pa = pp_smem;
  uint32_t* const pb = pa + (size_t)(s1 - s0 + 1) * S::AW;
  uint32_t* const red = pp_smem + P.red_off;
  load_planes<CFG>(pa, S::AW, A, min(16, P.m - strip * 16), 16, P.a_rs, P.r, P.a_cs, s0, s1 - s0 + 1);
  load_planes<CFG>(pb, S::BW, Bm, min(8, P.k - jt * 8), 8, P.b_cs, P.r, P.b_rs, u0, u1 - u0 + 1);
  __syncthreads();
  const int tl = warp % TC, sp = warp / TC, t = t0 + tl;
  int C[7][4];
#pragma unroll
  for (int q = 0; q < 7; ++q)
#pragma unroll
    for (int v = 0; v < 4; ++v) C[q][v] = 0;
  if (t < t_end) {
    const int sa = max(s0, t - (P.lb - 1)), sb = min(s1, t);
    for (int s = sa + sp; s <= sb; s += SS) {
      const uint32_t* a = pa + (size_t)(s - s0) * S::AW;
      const uint32_t* b = pb + (size_t)(t - s - u0) * S::BW;
      if constexpr (CFG == 0) {
        uint32_t H[4][2], Bh[4];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          H[l][0] = a[l * 64 + S::word(g, t4)];
          H[l][1] = a[l * 64 + S::word(g + 8, t4)];
          Bh[l] = b[l * 32 + S::word(g, t4)];
        }
#pragma unroll
        for (int q = 0; q < 7; ++q) {
          const int a0 = q < 4 ? 0 : q - 3, a1 = q < 4 ? q : 3;  // limbs a of the class, b = q - a
#pragma unroll
          for (int l = a0; l <= a1; l += 2) {
            const bool two = l + 1 <= a1;
            const uint32_t f[4] = {H[l][0], H[l][1], two ? H[two ? l + 1 : l][0] : 0u, two ? H[two ? l + 1 : l][1] : 0u};
            mma_u8(C[q], f, Bh[q - l], two ? Bh[two ? q - l - 1 : 0] : 0u);
          }
        }
      } else {
#pragma unroll
        for (int ks = 0; ks < CFG; ++ks) {
          uint32_t Af[4][4], Bf[4][2];
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            const uint32_t* al = a + l * 16 * S::KW;
            const uint32_t* bl = b + l * 8 * S::KW;
            Af[l][0] = al[S::word(g, 8 * ks + t4)];
            Af[l][1] = al[S::word(g + 8, 8 * ks + t4)];
            Af[l][2] = al[S::word(g, 8 * ks + t4 + 4)];
            Af[l][3] = al[S::word(g + 8, 8 * ks + t4 + 4)];
            Bf[l][0] = bl[S::word(g, 8 * ks + t4)];
            Bf[l][1] = bl[S::word(g, 8 * ks + t4 + 4)];
          }
#pragma unroll
          for (int l = 0; l < 4; ++l)
#pragma unroll
            for (int q = 0; q < 4; ++q) mma_u8(C[l + q], Af[l], Bf[q][0], Bf[q][1]);
        }
      }
    }
  }
  // join the limb classes: below 2^54 + 3 * 2^60.1, so one fold makes it fit the reduction
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    uint64_t x = (uint64_t)(uint32_t)C[0][v] + ((uint64_t)(uint32_t)C[1][v] << 8) + ((uint64_t)(uint32_t)C[2][v] << 16) +
                 ((uint64_t)(uint32_t)C[3][v] << 24);
    x += (uint64_t)(uint32_t)C[4][v] * P.w[0];
    x += (uint64_t)(uint32_t)C[5][v] * P.w[1];
    x += (uint64_t)(uint32_t)C[6][v] * P.w[2];
    red[((sp * 16 + g + 8 * (v >> 1)) * 8 + 2 * t4 + (v & 1)) * TC + tl] = redc(fold(x, M), M);
  }
  __syncthreads();
  for (int e = tid; e < TC * 128; e += kThreads) {
    const int c = e % TC, j = (e / TC) % 8, i = e / (TC * 8);
    uint32_t v = red[e];
#pragma unroll
    for (int q = 1; q < SS; ++q) v = addmod(v, red[q * TC * 128 + e], M.p);
    if (t0 + c < t_end && strip * 16 + i < P.m && jt * 8 + j < P.k)
      P.C[blockIdx.z * P.c_bs + (int64_t)(strip * 16 + i) * P.c_rs + (int64_t)(jt * 8 + j) * P.c_cs + (t0 + c - P.lo)] =
          redc_mul(v, P.r2, M);
  }
}

template <int CFG>
int launch(DirectProduct P, int nb, cudaStream_t s) {
  const int h = std::max(P.la, 1) - 1;
  P.red_off = (int)((size_t)(h + 1) * ProductShape<CFG>::AW + (size_t)(h + TC) * ProductShape<CFG>::BW);
  const dim3 grid((unsigned)((P.cnt + TC - 1) / TC), (unsigned)(((P.m + 15) / 16) * ((P.k + 7) / 8)), (unsigned)nb);
  direct_product_kernel<CFG><<<grid, kThreads, 4 * ((size_t)P.red_off + kRedWords), s>>>(P);
  RR_CUDA(cudaGetLastError());
  return RR_OK;
}

}  // namespace

// The largest degree of the left factor the direct product takes at inner
// dimension r: its planes fit shared memory, and beyond it the transform path,
// whose work grows as h log h and not as h^2, is faster.  One level lower is
// even for one generator (b = 16, d = 2^14, this line / lower: 88.6 / 90.7 ms) and
// better for batches, where the caller stops there.
int direct_product_max(int r) { return r <= 16 ? 128 : r <= 32 ? 64 : 32; }

int direct_product_prepare() {
  // the limits are per kernel, shared by every thread of the process: always the largest
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  RR_CUDA(cudaFuncSetAttribute(direct_product_kernel<0>, attr, (int)product_smem<0>(128)));
  RR_CUDA(cudaFuncSetAttribute(direct_product_kernel<1>, attr, (int)product_smem<1>(64)));
  RR_CUDA(cudaFuncSetAttribute(direct_product_kernel<2>, attr, (int)product_smem<2>(32)));
  return RR_OK;
}

int direct_product(DirectProduct P, int nb, cudaStream_t s) {
  if (P.la - 1 > direct_product_max(P.r))
    return fail(RR_EINVAL, "internal: direct product of degree %d at inner dimension %d", P.la - 1, P.r);
  P.w[0] = P.M.c32;
  P.w[1] = (uint32_t)((uint64_t)P.w[0] * 256 % P.M.p);
  P.w[2] = (uint32_t)((uint64_t)P.w[1] * 256 % P.M.p);
  P.r2 = (uint32_t)((uint64_t)P.M.r1 * P.M.r1 % P.M.p);
  if (P.r <= 16) return launch<0>(P, nb, s);
  if (P.r <= 32) return launch<1>(P, nb, s);
  return launch<2>(P, nb, s);
}

}  // namespace rr
