// krylov_gram.cuh -- lane layout of the block rows and the Gram accumulators
// shared by the Krylov kernels (krylov.cu, resident.cu).
#pragma once
#include "krylov_params.h"
#include "rr_device.cuh"

namespace rr {

// Threads of a warp split into RPW row slots of TPR threads; a thread owns
// LPT lanes of its row's block, as NV 128-bit words interleaved with the other
// threads of the slot: word v of thread `sub` is word v * TPR + sub of the row
// (lanes 4 (v TPR + sub) .. + 3).  So one warp load instruction reads TPR
// adjacent 16-byte words per row -- whole 32-byte sectors for B >= 8 -- and a
// gathered row costs the L1 the minimum of B / 8 sector accesses.
template <int B>
constexpr int kDefaultLpt = (B >= 16) ? 8 : 4;

template <int B, int L = kDefaultLpt<B>>
struct Shape {
  static constexpr int LPT = L;                   // lanes of the block per thread
  static constexpr int NV = LPT / 4;              // 128-bit words per thread per row
  static constexpr int TPR = B / LPT;             // threads per row
  static constexpr int RPW = 32 / TPR;            // rows per warp batch (slots)
  // block lane of this thread's lane l
  static __device__ __forceinline__ int lane_of(int sub, int l) { return 4 * ((l >> 2) * TPR + sub) + (l & 3); }
  // 128-bit word index within a row of this thread's word v
  static __device__ __forceinline__ int word_of(int sub, int v) { return v * TPR + sub; }
};

__device__ __forceinline__ void pair_of(int q, int B, int& i, int& j) {
  // q enumerates (i <= j) row-major: offset(i) = i*B - i*(i-1)/2
  i = 0;
  int off = 0;
  while (q >= off + (B - i)) {
    off += B - i;
    ++i;
  }
  j = i + (q - off);
}

__device__ __forceinline__ int pair_index(int i, int j, int B) { return i * B - i * (i - 1) / 2 + (j - i); }

// ---------------------------------------------------------------- Gram terms
// Both accumulators sum G[i][j] = sum over rows of gz[i] * gu[j] (i <= j) for
// the rows a warp processes, then add their residues into the CTA's red[].

// CUDA cores (B = 4): the batch is staged in shared memory and every lane
// accumulates a few (i, j) pairs over the staged rows.
template <int B, int L = kDefaultLpt<B>>
struct GramCore {
  static constexpr int LPT = Shape<B, L>::LPT, RPW = Shape<B, L>::RPW;
  static constexpr int NP = B * (B + 1) / 2, PPL = (NP + 31) / 32;
  static constexpr int kWords = 2 * RPW * B, kWordsSym = kWords;  // shared words per warp
  uint32_t* zs;  // [RPW][B]
  uint32_t* us;
  uint32_t pij[PPL];
  unsigned long long acc[PPL];

  __device__ __forceinline__ void init(uint32_t* w, int lane, bool = false) {
    zs = w;
    us = w + RPW * B;
#pragma unroll
    for (int t = 0; t < PPL; ++t) {
      const int q = lane + 32 * t;
      int i = 0, j = 0;
      if (q < NP) pair_of(q, B, i, j);
      pij[t] = ((uint32_t)i << 8) | (uint32_t)j;
      acc[t] = 0;
    }
  }
  __device__ __forceinline__ void add(const uint32_t (&gz)[LPT], const uint32_t (&gu)[LPT], int slot, int sub,
                                      int lane, const ModP& M, const uint32_t (&)[3]) {
#pragma unroll
    for (int l = 0; l < LPT; ++l) {
      zs[slot * B + Shape<B, L>::lane_of(sub, l)] = gz[l];
      us[slot * B + Shape<B, L>::lane_of(sub, l)] = gu[l];
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < PPL; ++t) {
      if (lane + 32 * t < NP) {
        const int i = pij[t] >> 8, j = pij[t] & 0xff;
        unsigned long long a = acc[t];
#pragma unroll
        for (int rr = 0; rr < RPW; ++rr) {
          a = mad_wide(zs[rr * B + i], us[rr * B + j], a);
          if ((rr % kFold) == kFold - 1) a = fold(a, M);
        }
        acc[t] = a;
      }
    }
    __syncwarp();
  }
  __device__ __forceinline__ void finish(int, int, int, const ModP&, const uint32_t (&)[3]) {}
  __device__ __forceinline__ void add_sym(const uint32_t (&gz)[LPT], int slot, int sub, int lane, const ModP& M,
                                          const uint32_t (&W)[3]) {
    add(gz, gz, slot, sub, lane, M, W);
  }
  __device__ __forceinline__ void finish_sym(int, int, int, const ModP&, const uint32_t (&)[3]) {}
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int t = 0; t < PPL; ++t) acc[t] = 0;
  }
  __device__ __forceinline__ void emit(unsigned long long* red, int lane, const ModP& M) {
#pragma unroll
    for (int t = 0; t < PPL; ++t) {
      const int q = lane + 32 * t;
      if (q < NP) atomicAdd(&red[q], (unsigned long long)reduce(acc[t], M));
    }
  }
  // the warp's sums as residues, part[i * B + j] for i <= j (others undefined)
  __device__ __forceinline__ void store(uint32_t* part, int lane, const ModP& M) {
#pragma unroll
    for (int t = 0; t < PPL; ++t) {
      const int q = lane + 32 * t;
      if (q < NP) part[(pij[t] >> 8) * B + (pij[t] & 0xff)] = reduce(acc[t], M);
    }
  }
};

// Tensor cores (B >= 8): exact integer Gram by byte limbs.  Residues are
// < 2^31, so z = sum_a z_a 256^a with bytes z_a, and
//   Z^T U = sum_{a,c} 256^{a+c} Z_a^T U_c.
// A warp stages 32 rows (one K tile) as byte planes P[limb][lane][row] in
// shared memory -- each row's four limbs are spread over four rows' words with
// a 4x4 byte transpose across lanes (two shuffles and two byte permutes) --
// then issues 16 m16n8k32 u8 MMAs per 16x8 output tile.  Per K tile a limb
// pair's product is < 32 * 255^2 < 2^21, so the shift classes s = a + c stay
// exact in int32; classes 0..3 are recombined exactly in 64 bits (< 2^48) and
// classes 4..6 are added with their weights 2^{8s} mod p.
template <int B, int L = kDefaultLpt<B>>
struct GramMma {
  static constexpr int LPT = Shape<B, L>::LPT, TPR = Shape<B, L>::TPR, RPW = Shape<B, L>::RPW;
  static constexpr int TB = 32 / RPW;           // batches per K tile
  static constexpr int BM = B < 16 ? 16 : B;    // rows of the M dimension (zero padded)
  static constexpr int MT = BM / 16, NT = B / 8;
  static constexpr int RS = 9;                  // words per (limb, lane) plane row: 32 bytes + 4 pad
  static constexpr int kPlane = 4 * BM * RS;    // words per plane set
  static constexpr int kWords = 2 * kPlane;     // shared words per warp
  static constexpr int kWordsSym = kPlane;      // with add_sym only
  uint32_t* pz;
  uint32_t* pu;
  unsigned long long acc[MT][NT][4];
  int bt;

  __device__ __forceinline__ void init(uint32_t* w, int lane, bool sym = false) {
    pz = w;
    pu = w + kPlane;
    for (int q = lane; q < (sym ? kWordsSym : kWords); q += 32) w[q] = 0;  // zero padding rows stay zero
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[mt][nt][v] = 0;
    bt = 0;
    __syncwarp();
  }

  // 4x4 byte transpose among the lanes holding rows 4q..4q+3 (lane distance
  // TPR): afterwards byte k of the word of the lane with row 4q+rho is limb
  // rho of the value of row 4q+k.
  __device__ __forceinline__ static uint32_t transpose4(uint32_t w, int rho) {
    uint32_t p = __shfl_xor_sync(0xffffffffu, w, TPR);
    w = (rho & 1) ? __byte_perm(p, w, 0x7351) : __byte_perm(w, p, 0x6240);
    p = __shfl_xor_sync(0xffffffffu, w, 2 * TPR);
    return (rho & 2) ? __byte_perm(p, w, 0x7632) : __byte_perm(w, p, 0x5410);
  }

  __device__ __forceinline__ void stage(const uint32_t (&gz)[LPT], const uint32_t (&gu)[LPT], int slot, int sub) {
    const int rho = slot & 3;
    const int word = (bt * RPW + (slot & ~3)) >> 2;  // 4-row group inside the K tile
#pragma unroll
    for (int l = 0; l < LPT; ++l) {
      const int i = Shape<B, L>::lane_of(sub, l);
      pz[(rho * BM + i) * RS + word] = transpose4(gz[l], rho);
      pu[(rho * BM + i) * RS + word] = transpose4(gu[l], rho);
    }
  }

  __device__ __forceinline__ void stage_sym(const uint32_t (&gz)[LPT], int slot, int sub) {
    const int rho = slot & 3;
    const int word = (bt * RPW + (slot & ~3)) >> 2;
#pragma unroll
    for (int l = 0; l < LPT; ++l) pz[(rho * BM + Shape<B, L>::lane_of(sub, l)) * RS + word] = transpose4(gz[l], rho);
  }

  // SYM: both factors are gz, and only its planes are staged (add_sym)
  template <bool SYM = false>
  __device__ __forceinline__ void flush(int lane, const ModP& M, const uint32_t (&W)[3]) {
    const uint32_t* const pv = SYM ? pz : pu;
    __syncwarp();
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      uint32_t A[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const uint32_t* r0 = pz + (a * BM + mt * 16 + g) * RS;
        const uint32_t* r1 = r0 + 8 * RS;
        A[a][0] = r0[t];
        A[a][1] = r1[t];
        A[a][2] = r0[t + 4];
        A[a][3] = r1[t + 4];
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        if (mt * 16 > nt * 8 + 7) continue;  // tile entirely below the diagonal
        uint32_t Bf[4][2];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t* r = pv + (c * BM + nt * 8 + g) * RS;
          Bf[c][0] = r[t];
          Bf[c][1] = r[t + 4];
        }
        uint64_t lo[4] = {0, 0, 0, 0};
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          int C[4] = {0, 0, 0, 0};
#pragma unroll
          for (int a = 0; a <= s; ++a) mma_u8(C, A[a], Bf[s - a][0], Bf[s - a][1]);
#pragma unroll
          for (int v = 0; v < 4; ++v) lo[v] += (uint64_t)(uint32_t)C[v] << (8 * s);
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[mt][nt][v] = fold(acc[mt][nt][v] + lo[v], M);
#pragma unroll
        for (int s = 4; s < 7; ++s) {
          int C[4] = {0, 0, 0, 0};
#pragma unroll
          for (int a = s - 3; a < 4; ++a) mma_u8(C, A[a], Bf[s - a][0], Bf[s - a][1]);
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[mt][nt][v] = mad_wide((uint32_t)C[v], W[s - 4], acc[mt][nt][v]);
        }
      }
    }
    __syncwarp();
  }

  __device__ __forceinline__ void add(const uint32_t (&gz)[LPT], const uint32_t (&gu)[LPT], int slot, int sub,
                                      int lane, const ModP& M, const uint32_t (&W)[3]) {
    stage(gz, gu, slot, sub);
    if (++bt == TB) {
      flush(lane, M, W);
      bt = 0;
    }
  }

  __device__ __forceinline__ void add_sym(const uint32_t (&gz)[LPT], int slot, int sub, int lane, const ModP& M,
                                          const uint32_t (&W)[3]) {
    stage_sym(gz, slot, sub);
    if (++bt == TB) {
      flush<true>(lane, M, W);
      bt = 0;
    }
  }
  __device__ __forceinline__ void finish_sym(int slot, int sub, int lane, const ModP& M, const uint32_t (&W)[3]) {
    if (bt == 0) return;
    uint32_t z[LPT];
#pragma unroll
    for (int l = 0; l < LPT; ++l) z[l] = 0;
    while (bt < TB) {
      stage_sym(z, slot, sub);
      ++bt;
    }
    flush<true>(lane, M, W);
    bt = 0;
  }

  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[mt][nt][v] = 0;
    bt = 0;
  }

  __device__ __forceinline__ void finish(int slot, int sub, int lane, const ModP& M, const uint32_t (&W)[3]) {
    if (bt == 0) return;
    uint32_t z[LPT];
#pragma unroll
    for (int l = 0; l < LPT; ++l) z[l] = 0;
    while (bt < TB) {  // zero the rows of the batches the tile did not get
      stage(z, z, slot, sub);
      ++bt;
    }
    flush(lane, M, W);
    bt = 0;
  }

  __device__ __forceinline__ void emit(unsigned long long* red, int lane, const ModP& M) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int i = mt * 16 + g + (v >= 2 ? 8 : 0);
          const int j = nt * 8 + 2 * t + (v & 1);
          if (i <= j && j < B) atomicAdd(&red[pair_index(i, j, B)], (unsigned long long)reduce(acc[mt][nt][v], M));
        }
  }
  // the warp's sums as residues, part[i * B + j] for i <= j (others undefined)
  __device__ __forceinline__ void store(uint32_t* part, int lane, const ModP& M) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (B >= 16 || v < 2)
            part[(mt * 16 + g + (v >= 2 ? 8 : 0)) * B + nt * 8 + 2 * t + (v & 1)] = reduce(acc[mt][nt][v], M);
  }
};

// Both Gram terms of an application from the rows of the even pass: the even
// term w' (x) w' and the odd term w (x) w' (w the block before the application),
// which together need one set of operands: no Gram work and no second block of
// multiply-adds in the odd pass.  Sums: [0, NP) odd, [NP, 2 NP) even.
template <int B, int L = kDefaultLpt<B>>
struct GramDual;

// B = 4: the lanes take the 10 pairs of either term.
template <>
struct GramDual<4, 4> {
  static constexpr int B = 4, RPW = 32, NP = 10;
  static constexpr int kWords = 2 * RPW * B;
  uint32_t *zs, *us;  // rows of w' and of w
  int pi, pj;
  unsigned long long acc;

  __device__ __forceinline__ void init(uint32_t* w, int lane) {
    zs = w;
    us = w + RPW * B;
    pi = pj = 0;
    if (lane < 2 * NP) pair_of(lane % NP, B, pi, pj);
    acc = 0;
  }
  __device__ __forceinline__ void add(const uint32_t (&w1)[4], const uint32_t (&w0)[4], int slot, int, int lane,
                                      const ModP& M, const uint32_t (&)[3]) {
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      zs[slot * B + l] = w1[l];
      us[slot * B + l] = w0[l];
    }
    __syncwarp();
    if (lane < 2 * NP) {
      const uint32_t* a = lane < NP ? us : zs;
#pragma unroll
      for (int rr = 0; rr < RPW; ++rr) {
        acc = mad_wide(a[rr * B + pi], zs[rr * B + pj], acc);
        if ((rr % kFold) == kFold - 1) acc = fold(acc, M);
      }
    }
    __syncwarp();
  }
  __device__ __forceinline__ void finish(int, int, int, const ModP&, const uint32_t (&)[3]) {}
  __device__ __forceinline__ void reset() { acc = 0; }
  __device__ __forceinline__ void emit(unsigned long long* red, int lane, const ModP& M) {
    if (lane < 2 * NP) atomicAdd(&red[lane], (unsigned long long)reduce(acc, M));
  }
};

// B = 8 on the tensor cores: the 16 rows of an MMA's A operand are the 8 lanes
// of w' and the 8 of w, so both terms take the products of one.
template <>
struct GramDual<8, 4> {
  static constexpr int B = 8, LPT = 4, TPR = 2, RPW = 16, TB = 2, RS = 9, NP = 36;
  static constexpr int kWords = 4 * 16 * RS;
  using Single = GramMma<8, 4>;
  uint32_t* pl;  // planes [limb][w' lanes 0..7, w lanes 8..15][RS]
  unsigned long long acc[4];
  int bt;

  __device__ __forceinline__ void init(uint32_t* w, int) {
    pl = w;
    reset();
  }
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[v] = 0;
    bt = 0;
  }
  __device__ __forceinline__ void stage(const uint32_t (&w1)[LPT], const uint32_t (&w0)[LPT], int slot, int sub) {
    const int rho = slot & 3, word = (bt * RPW + (slot & ~3)) >> 2;
#pragma unroll
    for (int l = 0; l < LPT; ++l) {
      const int i = Shape<B, 4>::lane_of(sub, l);
      pl[(rho * 16 + i) * RS + word] = Single::transpose4(w1[l], rho);
      pl[(rho * 16 + 8 + i) * RS + word] = Single::transpose4(w0[l], rho);
    }
  }
  __device__ __forceinline__ void flush(int lane, const ModP& M, const uint32_t (&W)[3]) {
    __syncwarp();
    const int g = lane >> 2, t = lane & 3;
    uint32_t A[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const uint32_t* r0 = pl + (a * 16 + g) * RS;
      A[a][0] = r0[t];
      A[a][1] = r0[8 * RS + t];
      A[a][2] = r0[t + 4];
      A[a][3] = r0[8 * RS + t + 4];
    }
    // the B operand's column g is lane g of w': the words of A's rows 0..7
    int C[7][4];
#pragma unroll
    for (int s = 0; s < 7; ++s)
#pragma unroll
      for (int v = 0; v < 4; ++v) C[s][v] = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) mma_u8(C[a + c], A[a], A[c][0], A[c][2]);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      uint64_t x = 0;
#pragma unroll
      for (int s = 0; s < 4; ++s) x += (uint64_t)(uint32_t)C[s][v] << (8 * s);
      uint64_t y = fold(acc[v] + x, M);
#pragma unroll
      for (int s = 4; s < 7; ++s) y = mad_wide((uint32_t)C[s][v], W[s - 4], y);
      acc[v] = y;
    }
    __syncwarp();
  }
  __device__ __forceinline__ void add(const uint32_t (&w1)[LPT], const uint32_t (&w0)[LPT], int slot, int sub, int lane,
                                      const ModP& M, const uint32_t (&W)[3]) {
    stage(w1, w0, slot, sub);
    if (++bt == TB) {
      flush(lane, M, W);
      bt = 0;
    }
  }
  __device__ __forceinline__ void finish(int slot, int sub, int lane, const ModP& M, const uint32_t (&W)[3]) {
    if (bt == 0) return;
    const uint32_t z[LPT] = {0, 0, 0, 0};
    stage(z, z, slot, sub);  // TB = 2: the one batch the tile did not get
    flush(lane, M, W);
    bt = 0;
  }
  // entry v of a lane: row g, column 2 t + (v & 1) of the even (v < 2) or odd term
  __device__ __forceinline__ void emit(unsigned long long* red, int lane, const ModP& M) {
    const int i = lane >> 2, j0 = 2 * (lane & 3);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int j = j0 + (v & 1);
      if (i <= j) atomicAdd(&red[(v < 2 ? NP : 0) + pair_index(i, j, B)], (unsigned long long)reduce(acc[v], M));
    }
  }
};

}  // namespace rr
