// pmleaf.cu -- one block of K order-1 leaves of the PM-basis and the block's
// basis, as one launch of a thread-block cluster per generator.
//
// Reference: src/sigma_basis.rs:348-416 (M_Basis), src/modular_linalg.rs:188-239
// (lsp_decomposition); the block equals the ordered product m_{K-1} ... m_0 of
// the order-1 bases (see pmbasis.cu).
//
// A leaf is a serial chain -- sort, at most n pivots, coefficient 0 of the next
// residual -- so it is bound by the latency of that chain on one SM, not by any
// throughput.  The cluster takes everything else off that SM:
//
//   rank 0            leaf CTA: the elimination (4 warps, 8 at n > 16)
//   ranks 1 .. nres   residual CTAs: cc columns each of the residual series
//   the others        basis CTAs: cc columns each of the block's basis
//
// Elimination (in place).  T = L^{-1} pi has only rank <= n non-trivial
// columns: one per pivot, plus the diagonal.  Once column cs has its pivot in
// row k its entries are zero in every later row, so its slot is reused for the
// column of L^{-1} that pivot k creates, and a step updates n columns instead
// of n + m.  Lane i of every warp holds row i (and row i + 32), warp w the
// CPW columns from CPW w on.  Rows are eliminated fraction-free,
//   row_i <- (piv row_i - a_i,cs row_k) R^{-1}   for i > k,
// so that no step needs an inverse; row i of the stored transform then carries
// the factor dg_i = its diagonal entry, and sigma accumulates it.
// The pivot is the first non-zero column of row k in the order of the
// unpivoted list (a pivot swaps places with the list's front).  Almost always
// that is the front itself, so a step publishes only the front column of the
// next step; when row k is zero there, the row is published and the first
// non-zero list position taken by one ballot.
//
// Coefficient 0 of the next residual: pivot rows take the eliminated row k as
// it stood when it became the pivot (no product at all); the other rows
// L^{-1} times coefficient 1, half a dot product per thread on the CUDA cores.
// Coefficient 1 comes from the residual CTAs, which have a whole elimination's
// time to compute it.
//
// Residual and basis updates,
//   R'[t - 1 + x_i][i] = T_i . R[t],   V'[t + x_i][i] = T_i . V[t]
// (x_i = 1 for pivot rows), run on the int8 tensor cores exactly: residues are
// < 2^31, so with byte limbs (T R) = sum over a, b of 256^(a+b) T_a R_b; the
// limb products of a class s = a + b summed over the inner dimension (<= 64)
// are at most (pairs of s) * 64 * 255^2 < 2^24, exact in int32, and
// C_1 2^8 + C_0, C_3 2^8 + C_2 and C_5 2^8 + C_4 stay below 2^32
// (4 * 64 * 255^2 * 257 < 2^32).  Classes 0..3 are joined in 64 bits (< 2^49),
// classes 4..6 added with weights 2^(8 s) mod p, and one Montgomery reduction
// gives (T R) R^{-1} (the sum is below p 2^32: the exact dot product is at most
// 64 p^2, so the low part is below p 2^32 for p < 2^26 and below 2^49
// otherwise; each weighted part is below 64 p^3 / 2^32 and below 2^63).
//
// Hand-offs: a finished transform goes from the leaf CTA's registers to the
// other CTAs' shared memory with st.async, and coefficient 1 comes back the
// same way; each message completes bytes on an mbarrier of its own (one per
// leaf), so no side needs a fence.  Every wait gives up after a limit (2 s by
// default) and sets *status = 3, after which the blocks that follow wait 0.2 ms at
// most; all CTAs meet in a cluster barrier before any of them exits.
// Measured (us per leaf, blocks of the largest K on one B200; before: one CTA
// per generator with 8 elimination and 8 update warps, then a second kernel for
// the block's basis -- 13.1 at n = 16 and 9.3 at n = 8, and the CUDA-core
// kernels at n = 32, 81): n = 16: 3.3, n = 8: 2.7, n = 1: 2.2, n = 32: 13.
// At n = 16 an elimination takes 3600 cycles (16 steps of 225: about 140 of
// issue, the barrier and the read), the transform, coefficient 0 and the
// barriers 1800; the largest residual and basis updates 5500, so the first and
// last leaves of a block wait for those.
#include <algorithm>
#include <type_traits>

#include "pm_mma.cuh"
#include "pmleaf.h"

namespace rr {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCluster = 8;      // portable cluster size
constexpr int kMaxLeaves = 64;
constexpr uint64_t kShortNs = 200000ull;
constexpr uint64_t kLandNs = 1000000ull;  // in which the messages in flight have long landed

// Words of the shared-memory regions; RL = rows per lane (m <= 32 RL), CPW =
// columns per elimination warp, EW = elimination warps (n <= CPW EW).
template <int RL, int CPW, int EW>
struct LeafShape {
  static constexpr int MP = 32 * RL;           // padded rows
  static constexpr int NP = EW * CPW;          // padded columns (pivot slots)
  static constexpr int KW = 8 * RL;            // words of a plane row (MP bytes)
  static constexpr int CC = 8 * RL;            // columns per residual or basis CTA
  static constexpr int NTC = CC / 8;
  // one coefficient as byte planes [limb][column][KW]; the padding puts the
  // same entry of neighbouring coefficients in different banks
  static constexpr int PW = 4 * CC * KW + 4;
  static constexpr int TW = 4 * MP * KW;       // T as byte planes [limb][row][KW]
  // a transform: L^{-1} slots [NP][MP], diagonal [MP], map [MP] (byte 0: source
  // row of row i; byte 1: slot of source row i, 255 = none), pivot-row mask (2)
  static constexpr int DIAG = NP * MP, MAP = DIAG + MP, MASK = MAP + MP, LW = MASK + 4;
  // transforms a residual or basis CTA holds: all of a block's, or (RL = 2,
  // where they are large) a ring whose slots it hands back
  static constexpr bool kRinged = RL > 1;
  static constexpr int slots(int K) { return kRinged ? 4 : K; }
  // row strides of coefficients 0 and 1: a warp's CPW columns are one load, and
  // the loads of a warp's rows fall in different banks
  static constexpr int RS0 = NP + CPW, RS1 = RS0;
  // offsets; the first regions are addressed by other CTAs
  static constexpr int OFF_BAR = 0;                         // mbarriers [kMaxLeaves + 1] (2 words each), used [8]
  static constexpr int OFF_USED = OFF_BAR + 2 * (kMaxLeaves + 2);
  static constexpr int OFF_SIG = OFF_USED + 8;              // sigma [MP]
  static constexpr int OFF_R1 = OFF_SIG + MP;               // leaf CTA: R1 [2][MP + 1][RS1]
  static constexpr int PWARPS = NP < 8 ? NP : 8;            // warps that form coefficient 0
  static constexpr int R1W = (MP + 1) * RS1;                // with a zero row at the end
  static constexpr int OFF_R0 = OFF_R1 + 2 * R1W;           // R0 [2][MP][RS0]
  static constexpr int OFF_FB = OFF_R0 + 2 * MP * RS0;      // front column [2][MP]
  static constexpr int OFF_ROW = OFF_FB + 2 * MP;           // published row [2][32]
  static constexpr int OFF_SORT = OFF_ROW + 64;             // small arrays (LeafScratch)
  static constexpr int OFF_L = (OFF_SORT + 4 * MP + 36 + MP + 6 * MP + 3) & ~3;  // slots, diagonal [NP + 1][MP]
  static constexpr int LEAF_WORDS = OFF_L + (NP + 1) * MP;
  static constexpr int OFF_T = (OFF_R1 + 3) & ~3;           // other CTAs: T planes [2]
  static constexpr int OFF_RING = OFF_T + 2 * TW;           // transforms [slots][LW]
  static constexpr size_t smem_bytes(int K) {
    const size_t upd = (size_t)OFF_RING + (size_t)slots(K) * LW + (size_t)2 * (K + 1) * PW;
    return 4 * (LEAF_WORDS > upd ? LEAF_WORDS : upd);
  }
  static_assert(LW % 4 == 0 && OFF_RING % 4 == 0 && OFF_BAR % 2 == 0 && MAP % 4 == 0, "alignment");
};

// the same address in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(p)), "r"(rank));
  return r;
}
// a 4-byte store into another CTA that completes 4 bytes on that CTA's mbarrier
__device__ __forceinline__ void st_async(uint32_t a, uint32_t v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(a), "r"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async4(uint32_t a, uint4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.u32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(a),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_peer_release(uint32_t a, uint32_t v) {
  asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// mbarrier `q` of this CTA: armed for one message of `bytes` bytes
__device__ __forceinline__ void bar_arm(uint32_t* sm, int q, uint32_t bytes) {
  const uint32_t a = smem_addr(sm + 2 * q);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(a) : "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t a) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], 0;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}\n"
      : "=r"(done)
      : "r"(a)
      : "memory");
  return done != 0;
}
// Waits for the message of mbarrier q; gives up after wait_ns, once another
// wait of this CTA did, or soon if one of an earlier block did, whose basis is then
// not there (looked up after kShortNs only: no wait of a running block takes so long).
__device__ __forceinline__ bool bar_wait(uint32_t* sm, int q, volatile int* abort, const LeafBlock& P) {
  const uint32_t a = smem_addr(sm + 2 * q);
  if (bar_try(a)) return true;
  const uint64_t t0 = now_ns();
  do {
    if (bar_try(a)) return true;
    if (*abort) return false;
  } while (now_ns() - t0 <= kShortNs);
  while (now_ns() - t0 <= P.wait_ns && *(volatile int*)P.status != 3) {
    if (bar_try(a)) return true;
    if (*abort) return false;
  }
  *abort = 1;
  atomicExch(P.status, 3);
  return false;
}

// *p = v where `on` holds, as one predicated store
__device__ __forceinline__ void st_shared_if(uint32_t* p, uint32_t v, bool on) {
  asm volatile("{\n\t.reg .pred P1;\n\tsetp.ne.u32 P1, %2, 0;\n\t@P1 st.shared.u32 [%0], %1;\n\t}\n" ::"r"(smem_addr(p)),
               "r"(v), "r"((uint32_t)on)
               : "memory");
}

template <int EW>
__device__ __forceinline__ void elim_bar() {
  asm volatile("bar.sync 1, %0;" ::"n"(EW * 32) : "memory");
}

// a^{-1} R mod p (p prime): a^(p-2) on Montgomery representatives; the square
// and the product of a step are independent.
__device__ uint32_t inverse_r(uint32_t a, const ModP& M) {
  uint32_t b = redc_mul(a, mulmod(M.r1, M.r1, M), M), r = M.r1;
  for (uint32_t e = M.p - 2; e; e >>= 1) {
    const uint32_t rb = redc_mul(r, b, M);
    r = (e & 1) ? rb : r;
    b = redc_mul(b, b, M);
  }
  return r;
}

// CPW adjacent words in one load
template <int CPW>
__device__ __forceinline__ void load_words(const uint32_t* p, uint32_t (&v)[CPW]) {
  if constexpr (CPW == 4) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else if constexpr (CPW == 2) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    v[0] = q.x, v[1] = q.y;
  } else {
    v[0] = *p;
  }
}

// Byte offset of (column, row) in a limb plane.
template <int RL>
__device__ __forceinline__ int plane_byte(int col, int row) {
  return 4 * plane_word<RL>(col, row >> 2) + (row & 3);
}
template <int RL>
__device__ __forceinline__ void plane_store(uint32_t* coeff, int byte, uint32_t v) {
  unsigned char* b = reinterpret_cast<unsigned char*>(coeff) + byte;
#pragma unroll
  for (int l = 0; l < 4; ++l) b[4 * l * (8 * RL) * (8 * RL)] = (unsigned char)(v >> (8 * l));
}
template <int RL>
__device__ __forceinline__ uint32_t plane_load(const uint32_t* coeff, int byte) {
  const unsigned char* b = reinterpret_cast<const unsigned char*>(coeff) + byte;
  uint32_t v = 0;
#pragma unroll
  for (int l = 0; l < 4; ++l) v |= (uint32_t)b[4 * l * (8 * RL) * (8 * RL)] << (8 * l);
  return v;
}

// Four 16 x 8 byte matrices in the accumulator layout (rows g and g + 8,
// columns 2 t4 and 2 t4 + 1 of a thread), stored transposed: lane 8 l + c gives
// the address of the 16 bytes of column c of matrix l.
__device__ __forceinline__ void stmatrix_u8(uint32_t addr, const uint32_t (&w)[4]) {
  asm volatile("stmatrix.sync.aligned.m16n8.x4.trans.shared.b8 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]),
               "r"(w[2]), "r"(w[3])
               : "memory");
}

// The fragments of T's rows 16 mt .. 16 mt + 15.
template <int RL>
__device__ __forceinline__ void load_rows(const uint32_t* Tp, int mt, int g, int t4, uint32_t (&A)[RL][4][4]) {
  constexpr int MP = 32 * RL, KW = 8 * RL;
  const int r0 = mt * 16 + g, r1 = r0 + 8;
#pragma unroll
  for (int ks = 0; ks < RL; ++ks)
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t* tp = Tp + l * MP * KW;
      A[ks][l][0] = tp[plane_word<RL>(r0, 8 * ks + t4)];
      A[ks][l][1] = tp[plane_word<RL>(r1, 8 * ks + t4)];
      A[ks][l][2] = tp[plane_word<RL>(r0, 8 * ks + t4 + 4)];
      A[ks][l][3] = tp[plane_word<RL>(r1, 8 * ks + t4 + 4)];
    }
}

// Joins the limb classes of a tile: val = redc(sum of C_s 2^(8 s)).
__device__ __forceinline__ void join_classes(const int (&C)[7][4], const uint32_t (&Wt)[3], const ModP& M,
                                             uint32_t (&val)[4]) {
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    uint64_t x = (uint64_t)((uint32_t)C[5][v] * 256u + (uint32_t)C[4][v]) * Wt[0] +
                 (uint32_t)((uint32_t)C[1][v] * 256u + (uint32_t)C[0][v]);
    x += (uint64_t)((uint32_t)C[3][v] * 256u + (uint32_t)C[2][v]) * Wt[2];  // 2^16: one instruction, where a shift takes four
    x += (uint64_t)(uint32_t)C[6][v] * Wt[1];
    val[v] = redc(x, M);
  }
}

// A strip of 16 rows of T times columns 8 nt .. 8 nt + 7 of one coefficient
// (planes), over KS k-steps of 32 from word `w0` of the plane rows on: val[v] =
// redc of the product at row 16 mt + g + 8 (v >> 1), column 8 nt + 2 t4 + (v & 1).
template <int RL, int KS>
__device__ __forceinline__ void tile_product(const uint32_t (&A)[KS][4][4], const uint32_t* V, int w0, int nt, int g,
                                             int t4, const uint32_t (&Wt)[3], const ModP& M, uint32_t (&val)[4]) {
  constexpr int CC = 8 * RL, KW = 8 * RL;
  int C[7][4];
  const int col = nt * 8 + g;
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    uint32_t Bf[4][2];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t* vp = V + l * CC * KW;
      Bf[l][0] = vp[plane_word<RL>(col, w0 + 8 * ks + t4)];
      Bf[l][1] = vp[plane_word<RL>(col, w0 + 8 * ks + t4 + 4)];
    }
#pragma unroll
    for (int l = 0; l < 4; ++l)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (ks == 0 && (l == 0 || r == 3)) mma_u8_first(C[l + r], A[ks][l], Bf[r][0], Bf[r][1]);
        else mma_u8(C[l + r], A[ks][l], Bf[r][0], Bf[r][1]);
      }
  }
  join_classes(C, Wt, M, val);
}

// The same where the strip is zero but for 16 source rows (plane words w0 ..
// w0 + 3): two limb pairs share one k-step, 10 products instead of 16.
// A[l] = limb l of rows g and g + 8.
__device__ __forceinline__ void tile_product_half(const uint32_t (&A)[4][2], const uint32_t* V, int w0, int nt, int g,
                                                  int t4, const uint32_t (&Wt)[3], const ModP& M, uint32_t (&val)[4]) {
  uint32_t B[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) B[l] = V[l * 64 + plane_word<1>(nt * 8 + g, w0 + t4)];
  int C[7][4];
#pragma unroll
  for (int s = 0; s < 7; ++s) {
    const int a0 = s < 4 ? 0 : s - 3, a1 = s < 4 ? s : 3;  // limbs a of the class, b = s - a
#pragma unroll
    for (int a = a0; a <= a1; a += 2) {
      const bool two = a + 1 <= a1;
      const uint32_t f[4] = {A[a][0], A[a][1], two ? A[two ? a + 1 : a][0] : 0u, two ? A[two ? a + 1 : a][1] : 0u};
      const uint32_t b0 = B[s - a], b1 = two ? B[two ? s - a - 1 : 0] : 0u;
      if (a == a0) mma_u8_first(C[s], f, b0, b1);
      else mma_u8(C[s], f, b0, b1);
    }
  }
  join_classes(C, Wt, M, val);
}

template <int CPW>
__device__ __forceinline__ uint32_t pick(const uint32_t (&a)[CPW], int cl) {  // a[cl], cl uniform
  uint32_t v = a[0];
#pragma unroll
  for (int j = 1; j < CPW; ++j) v = cl == j ? a[j] : v;
  return v;
}
// a[r] of a per-row pair, r uniform
template <int RL>
__device__ __forceinline__ uint32_t of_row(uint32_t lo, uint32_t hi, int r) {
  return RL > 1 && r ? hi : lo;
}

// ---------------------------------------------------------------- leaf CTA
// Warps 0 .. EW-1 eliminate and form coefficient 0 of the next residual;
// between two eliminations warps 8 .. 13 send the transform to one CTA each and
// warp 14 sorts; warp 15 waits for coefficient 1 during the elimination.
constexpr int kSendWarp = 8, kSortWarp = 14, kWaitWarp = 15;

template <int RL, int CPW, int EW>
struct LeafScratch {
  using S = LeafShape<RL, CPW, EW>;
  using Mask = typename std::conditional<RL == 1, uint32_t, unsigned long long>::type;  // a bit per row
  uint32_t *R1, *R0, *fb, *rowbuf, *L, *sig, *mask;
  int *perm, *del, *row, *src, *nplist, *slot;
  __device__ explicit LeafScratch(uint32_t* sm) {
    constexpr int MP = S::MP;
    R1 = sm + S::OFF_R1;
    R0 = sm + S::OFF_R0;
    fb = sm + S::OFF_FB;
    rowbuf = sm + S::OFF_ROW;
    L = sm + S::OFF_L;           // [NP][MP] columns of L^{-1} by pivot number, then the diagonal [MP]
    uint32_t* q = sm + S::OFF_SORT;
    sig = q, q += MP;            // row scales by row
    perm = (int*)q, q += MP;     // source row by sorted position (next leaf)
    del = (int*)q, q += MP;      // delta by sorted position
    row = (int*)q, q += MP;      // source row by sorted position (this leaf), times RS1
    src = (int*)q, q += 32;      // source row of pivot number r, times RS1
    mask = q, q += 4;            // pivot rows (2 words), number of pivots
    nplist = (int*)q, q += MP;   // the rows without a pivot
    slot = (int*)q;              // per sender: pivot number of a source row
  }
};

// Coefficient 0 of the nn rows without a pivot: L^{-1} times coefficient 1.
// Warp w takes PC columns; lanes l and l + 16 share an output, each taking
// every other pivot.
template <int RL, int CPW, int EW>
__device__ __forceinline__ void leaf_products(const LeafBlock& P, const LeafScratch<RL, CPW, EW>& X, int leaf, int nn) {
  using S = LeafShape<RL, CPW, EW>;
  constexpr int MP = S::MP, NP = S::NP, PC = NP / S::PWARPS;
  const ModP M = P.M;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4;
  const uint32_t* R1c = X.R1 + (leaf & 1) * S::R1W + PC * warp;
  uint32_t* R0n = X.R0 + ((leaf + 1) & 1) * MP * S::RS0 + PC * warp;
  int off[NP / 2];
#pragma unroll
  for (int q = 0; q < NP / 2; ++q) off[q] = X.src[2 * q + half];
  for (int j0 = 0; j0 < nn; j0 += 16) {
    const int j = j0 + (lane & 15);
    const int i = j < nn ? X.nplist[j] : 0;
    const uint32_t* Lp = X.L + half * MP + i;
    uint32_t l[NP / 2], r1[NP / 2][PC], r1d[PC];
#pragma unroll
    for (int q = 0; q < NP / 2; ++q) {
      l[q] = Lp[2 * q * MP];
      load_words<PC>(R1c + off[q], r1[q]);
    }
    const uint32_t d = half == 0 ? X.L[NP * MP + i] : 0u;
    load_words<PC>(R1c + X.row[i], r1d);
    uint64_t x[PC];
#pragma unroll
    for (int cl = 0; cl < PC; ++cl) {
      x[cl] = 0;
#pragma unroll
      for (int q = 0; q < NP / 2; ++q) {
        x[cl] += (uint64_t)l[q] * r1[q][cl];
        if ((q & 3) == 3) x[cl] = fold(x[cl], M);  // four products fit between folds for every p < 2^31
      }
      x[cl] += (uint64_t)d * r1d[cl];
    }
#pragma unroll
    for (int cl = 0; cl < PC; ++cl) {
      uint32_t y = redc(fold(x[cl], M), M);
      y = addmod(y, __shfl_xor_sync(0xffffffffu, y, 16), M.p);
      if (j < nn && half == 0) R0n[i * S::RS0 + cl] = y;
    }
  }
}

template <int RL, int CPW, int EW>
__device__ void leaf_eliminate(const LeafBlock& P, uint32_t* sm, const volatile int* s_ok) {
  using S = LeafShape<RL, CPW, EW>;
  using Mask = typename LeafScratch<RL, CPW, EW>::Mask;
  constexpr int MP = S::MP, NP = S::NP, RS0 = S::RS0, RS1 = S::RS1;
  const LeafScratch<RL, CPW, EW> X(sm);
  const int m = P.m, n = P.n, K = P.K;
  const ModP M = P.M;
  const uint32_t p = M.p;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t R2 = mulmod(M.r1, M.r1, M);  // R^2 mod p
  int rowpar = 0;
  for (int leaf = 0; leaf < K; ++leaf) {
    const uint32_t* R0c = X.R0 + (leaf & 1) * MP * RS0;
    uint32_t* R0n = X.R0 + ((leaf + 1) & 1) * MP * RS0;
    // rows of pi r (the sorted order) and the first front column, column 0
    uint32_t a[RL][CPW], dg[RL], f[RL], ak[CPW];
    uint32_t sk[CPW];  // product of the pivots before this column's own; 0 = not pivoted yet
    int perm[RL];
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      perm[r] = X.perm[lane + 32 * r];
      const uint32_t* row = R0c + perm[r] * RS0;
      load_words<CPW>(row + CPW * warp, a[r]);  // columns >= n and rows >= m are zero
      f[r] = row[0];
      dg[r] = 1;
    }
#pragma unroll
    for (int cl = 0; cl < CPW; ++cl) {
      sk[cl] = 0;
      ak[cl] = __shfl_sync(0xffffffffu, a[0][cl], 0);
    }
    int lst = lane;    // column at list position `lane`: the pivoted ones in order, then the unpivoted
    int prow = lane;   // row of pivot number `lane`
    uint32_t s = 1;    // product of the pivots so far (with their R^{-1})
    int rank = 0;
    uint32_t piv = __shfl_sync(0xffffffffu, f[0], 0);
    // As long as row j has its pivot in column j (every step of a generic
    // leaf).  The chain of a step is one Montgomery product, the store of the
    // next front column, the barrier and the read; the other columns are
    // updated while that read is in flight.  Unrolled over the columns of one
    // warp, so that registers are known to the compiler, and no further: code
    // that runs once per leaf waits for its instructions.
    for (int w = 0; w < EW && rank < n && piv != 0; ++w) {
#pragma unroll
      for (int c = 0; c < CPW; ++c) {
        const int j = CPW * w + c;
        constexpr int kEven = CPW % 2 == 0;
        const int par = kEven ? (c + 1) & 1 : (j + 1) & 1;  // buffer of the next front column
        const int c1 = (c + 1) % CPW;
        const bool own = warp == w, more = j + 1 < n;
        const bool own_next = c + 1 < CPW ? own : warp == w + 1;
        uint32_t f2[RL], piv2 = 0;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const uint32_t nv = redc2(piv, a[r][c1], p - f[r], ak[c1], M);
          if (r > 0 || lane > j) a[r][c1] = nv;
          st_shared_if(X.fb + par * MP + lane + 32 * r, a[r][c1], own_next && more);
          f2[r] = 0;
        }
        if (more) {
          elim_bar<EW>();
#pragma unroll
          for (int r = 0; r < RL; ++r) f2[r] = X.fb[par * MP + lane + 32 * r];
          piv2 = X.fb[par * MP + j + 1];
        }
#pragma unroll
        for (int cl = 0; cl < CPW; ++cl) {
          if (cl == c1) continue;
#pragma unroll
          for (int r = 0; r < RL; ++r) {
            const uint32_t nv = redc2(piv, a[r][cl], p - f[r], ak[cl], M);
            if (r > 0 || lane > j) a[r][cl] = nv;
          }
        }
        // in the warp of the pivot column: its part of the pivot rows, then the
        // column of L^{-1} without its factor s_k R^{-1}
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const bool below = r > 0 || lane > j;
          st_shared_if(R0n + (lane + 32 * r) * RS0 + j, below ? 0u : f[r], own);
          const uint32_t nf = f[r] ? p - f[r] : 0u;
          const uint32_t nv = below ? nf : (lane == j ? M.r1 : 0u);
          a[r][c] = own ? nv : a[r][c];
        }
        sk[c] = own ? s : sk[c];
        s = redc_mul(piv, s, M);
#pragma unroll
        for (int r = 0; r < RL; ++r)
          if (r > 0 || lane > j) dg[r] = s;
        rank = j + 1;
        piv = piv2;
        if (!more) break;
#pragma unroll
        for (int cl = 0; cl < CPW; ++cl) ak[cl] = __shfl_sync(0xffffffffu, a[0][cl], (j + 1) & 31);
#pragma unroll
        for (int r = 0; r < RL; ++r) f[r] = f2[r];
        if (piv == 0) break;
      }
    }
    int number[CPW];  // pivot number of this warp's columns
#pragma unroll
    for (int cl = 0; cl < CPW; ++cl) number[cl] = CPW * warp + cl;
    Mask pm = ((Mask)1 << (rank & 31)) - 1;  // pivot rows
    if (RL > 1 && rank == 32) pm = (Mask)0xffffffffu;
    int par = rank & 1, k = rank, cs = rank;
    // From the first row without a pivot in the front column on.  Written
    // without branches but for the loop's own: one not taken costs 25 cycles.
    while (rank < n) {
      if (piv == 0) {  // row k is zero in the front column: look at the others
        const int kl = k & 31, kr = RL > 1 ? k >> 5 : 0;
        if (lane == kl) {
#pragma unroll
          for (int cl = 0; cl < CPW; ++cl) {
            const int c = CPW * warp + cl;
            if (c < n) X.rowbuf[rowpar * 32 + c] = sk[cl] == 0 ? of_row<RL>(a[0][cl], a[RL - 1][cl], kr) : 0u;
          }
        }
        __syncwarp();  // a warp must arrive at a named barrier as one
        elim_bar<EW>();
        const uint32_t v = lane >= rank && lane < n ? X.rowbuf[rowpar * 32 + lst] : 0u;
        rowpar ^= 1;
        const uint32_t hit = __ballot_sync(0xffffffffu, v != 0);
        if (hit == 0) {  // no pivot in row k (the same decision in every warp)
          if (++k == m) break;
          const int jl = k & 31, jr = RL > 1 ? k >> 5 : 0;
          piv = __shfl_sync(0xffffffffu, of_row<RL>(f[0], f[RL - 1], jr), jl);
#pragma unroll
          for (int cl = 0; cl < CPW; ++cl)
            ak[cl] = __shfl_sync(0xffffffffu, of_row<RL>(a[0][cl], a[RL - 1][cl], jr), jl);
          continue;
        }
        const int ts = __ffs(hit) - 1;
        const int front = cs;
        cs = __shfl_sync(0xffffffffu, lst, ts);
        if (lane == ts) lst = front;
        if (lane == rank) lst = cs;
        par ^= 1;
        if (cs / CPW == warp) {
#pragma unroll
          for (int r = 0; r < RL; ++r) X.fb[par * MP + lane + 32 * r] = pick<CPW>(a[r], cs % CPW);
        }
        __syncwarp();
        elim_bar<EW>();
#pragma unroll
        for (int r = 0; r < RL; ++r) f[r] = X.fb[par * MP + lane + 32 * r];
        piv = X.fb[par * MP + k];
      }
      const int next = __shfl_sync(0xffffffffu, lst, rank + 1);  // the next front column (if any is left)
      const bool last = rank + 1 == n || k + 1 == m;
      par ^= 1;
#pragma unroll
      for (int cl = 0; cl < CPW; ++cl)
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const uint32_t nv = redc2(piv, a[r][cl], p - f[r], ak[cl], M);
          if (lane + 32 * r > k) a[r][cl] = nv;
        }
      {
        const bool pub = !last && next / CPW == warp;
#pragma unroll
        for (int r = 0; r < RL; ++r)
          st_shared_if(X.fb + par * MP + lane + 32 * r, pick<CPW>(a[r], next % CPW), pub);
      }
      const bool own = cs / CPW == warp;
      if (RL == 1 || own) {
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const int i = lane + 32 * r;
          st_shared_if(R0n + i * RS0 + cs, i <= k ? f[r] : 0u, own);
          const uint32_t nv = i > k ? (f[r] ? p - f[r] : 0u) : (i == k ? M.r1 : 0u);
#pragma unroll
          for (int cl = 0; cl < CPW; ++cl) a[r][cl] = own && cl == cs % CPW ? nv : a[r][cl];
        }
#pragma unroll
        for (int cl = 0; cl < CPW; ++cl) {
          sk[cl] = own && cl == cs % CPW ? s : sk[cl];
          number[cl] = own && cl == cs % CPW ? rank : number[cl];
        }
      }
      s = redc_mul(piv, s, M);
#pragma unroll
      for (int r = 0; r < RL; ++r) dg[r] = lane + 32 * r > k ? s : dg[r];
      prow = lane == rank ? k : prow;
      pm |= (Mask)1 << k;
      ++rank;
      if (last) break;
      ++k;
      cs = next;
#pragma unroll
      for (int cl = 0; cl < CPW; ++cl)
        ak[cl] = __shfl_sync(0xffffffffu, of_row<RL>(a[0][cl], a[RL - 1][cl], RL > 1 ? k >> 5 : 0), k & 31);
      elim_bar<EW>();
#pragma unroll
      for (int r = 0; r < RL; ++r) f[r] = X.fb[par * MP + lane + 32 * r];
      piv = X.fb[par * MP + k];
    }
    // The transform.  Pivot rows of coefficient 0 are the eliminated rows
    // themselves, so their rows of T take another factor R, which makes up for
    // the R^{-1} of the products with the other coefficients.
    int src = __shfl_sync(0xffffffffu, perm[0], prow & 31);  // source row of pivot number `lane`
    if (RL > 1) {
      const int y = __shfl_sync(0xffffffffu, perm[RL - 1], prow & 31);
      src = prow >= 32 ? y : src;
    }
    bool isp[RL];
#pragma unroll
    for (int r = 0; r < RL; ++r) isp[r] = (pm >> (lane + 32 * r)) & 1;
#pragma unroll
    for (int cl = 0; cl < CPW; ++cl) {
      const uint32_t skr = redc_mul(sk[cl], R2, M);
      const bool done = sk[cl] != 0;
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const int i = lane + 32 * r;
        st_shared_if(X.L + number[cl] * MP + i, redc_mul(a[r][cl], isp[r] ? skr : sk[cl], M), done);
        st_shared_if(R0n + i * RS0 + CPW * warp + cl, a[r][cl], !done);  // pivot rows; the others are formed below
      }
    }
    if (warp == 0) {
      X.src[lane] = (lane < rank ? src : MP) * RS1;  // past the last pivot: the zero row
      if (lane < 3) X.mask[lane] = lane == 0 ? (uint32_t)pm : lane == 1 ? (uint32_t)((unsigned long long)pm >> 32) : rank;
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const int i = lane + 32 * r;
        X.row[i] = perm[r] * RS1;
        X.L[NP * MP + i] = i < m ? (isp[r] ? redc_mul(dg[r], R2, M) : dg[r]) : 0u;
      }
    } else if (warp == 1) {
      bool zero = false;
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const int i = lane + 32 * r;
        const Mask lt = ((Mask)1 << i) - 1;
        st_shared_if(reinterpret_cast<uint32_t*>(X.nplist) +
                         (RL == 1 ? __popc(~(uint32_t)pm & (uint32_t)lt) : __popcll(~pm & lt)),
                     (uint32_t)i, i < m && !isp[r]);
        zero = zero || (i < m && dg[r] == 0);
      }
      if (__any_sync(0xffffffffu, zero)) atomicExch(P.status, 2);
    }
    __syncthreads();  // the transform is complete, and coefficient 1 is here
    if (leaf + 1 == K || !*s_ok) return;
    if (warp < S::PWARPS) leaf_products<RL, CPW, EW>(P, X, leaf, m - rank);
    __syncthreads();  // coefficient 0 and the next order are complete
  }
}

template <int RL, int CPW, int EW>
__device__ void leaf_help(const LeafBlock& P, uint32_t* sm, volatile int* s_abort, volatile int* s_ok) {
  using S = LeafShape<RL, CPW, EW>;
  using Mask = typename LeafScratch<RL, CPW, EW>::Mask;
  constexpr int MP = S::MP, NP = S::NP;
  const LeafScratch<RL, CPW, EW> X(sm);
  const int m = P.m, n = P.n, K = P.K, csize = 1 + P.nres + P.nbas;
  const ModP M = P.M;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t dbase = P.delta[0];
  const int peer = warp - kSendWarp + 1;  // a sender's CTA
  const bool sender = peer >= 1 && peer < csize;
  for (int leaf = 0; leaf < K; ++leaf) {
    // during the elimination: what does not depend on its pivots
    int perm[RL], del[RL];
    Mask heads = 0;     // rows where a group of equal delta starts
    uint32_t sig[RL];
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      const int i = lane + 32 * r;
      perm[r] = X.perm[i];
      del[r] = X.del[i];
      sig[r] = X.sig[perm[r]];
      const int prev = i > 0 ? X.del[i - 1] : 0;
      heads |= (Mask)__ballot_sync(0xffffffffu, i < m && (i == 0 || prev != del[r])) << (32 * (r & (RL - 1)));
      if (sender) X.slot[(peer - 1) * MP + i] = 255;
    }
    if (warp == kWaitWarp && leaf > 0 && leaf + 1 < K) {
      const bool ok = bar_wait(sm, leaf - 1, s_abort, P);
      if (!__all_sync(0xffffffffu, ok) && lane == 0) *s_ok = 0;
    }
    if (S::kRinged && leaf >= S::slots(K) && sender) {
      // the ring slot this transform goes to (handed back long ago)
      const uint64_t t0 = now_ns();
      while (ld_acquire(sm + S::OFF_USED + peer) < (uint32_t)(leaf - S::slots(K) + 1)) {
        if (*s_abort || now_ns() - t0 > P.wait_ns) {
          *s_abort = 1;
          atomicExch(P.status, 3);
          *s_ok = 0;
          break;
        }
      }
      __syncwarp();
    }
    __syncthreads();
    if (!*s_ok) return;
    const Mask pm = (Mask)(((unsigned long long)X.mask[1] << 32) | X.mask[0]);
    // (a residual CTA has nothing to do in the last two leaves)
    if (sender && peer >= (leaf < K - 2 ? 1 : 1 + P.nres)) {
      const uint32_t bar = peer_addr(sm + 2 * leaf, peer);
      const uint32_t to = peer_addr(sm + S::OFF_RING + (leaf % S::slots(K)) * S::LW, peer);
      const uint4* from = reinterpret_cast<const uint4*>(X.L);
#pragma unroll
      for (int u = 0; u < NP * MP / 128; ++u) {
        const int e = lane + 32 * u;
        if (4 * e < n * MP) st_async4(to + 16 * e, from[e], bar);
      }
      if (lane < MP / 4) st_async4(to + 16 * (S::DIAG / 4 + lane), from[NP * MP / 4 + lane], bar);
      int* slot = X.slot + (peer - 1) * MP;
      if (lane < (int)X.mask[2]) slot[X.src[lane] / S::RS1] = lane;
      __syncwarp();
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const int i = lane + 32 * r;
        st_async(to + 4 * (S::MAP + i), (uint32_t)(perm[r] | (slot[i] << 8)), bar);
      }
      if (lane < 2) st_async(to + 4 * (S::MASK + lane), X.mask[lane], bar);
    }
    if (warp == kSortWarp) {
      // delta and sigma in the new order of rows; the next leaf's stable sort:
      // within a group of equal delta the rows that kept it come first
      uint32_t sg[RL];
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const int i = lane + 32 * r;
        int to = i, dl = 0;
        sg[r] = 0;
        if (i < m) {
          const bool isp = (pm >> i) & 1;
          const Mask lt = ((Mask)1 << i) - 1, upto = (lt << 1) | 1;
          const Mask later = heads & ~upto, below = heads & upto;
          const int start = RL == 1 ? 31 - __clz((int)(uint32_t)below) : 63 - __clzll((long long)below);
          const Mask end_mask = later ? (later & (~later + 1)) - 1 : (Mask) ~(Mask)0;  // rows before the next group
          const Mask grp = end_mask & ~(((Mask)1 << start) - 1);
          const Mask kept = grp & ~pm & (m == MP ? (Mask) ~(Mask)0 : ((Mask)1 << m) - 1);
          if (leaf + 1 < K) {
            if (RL == 1)
              to = start + (isp ? __popc((uint32_t)kept) + __popc((uint32_t)(grp & pm & lt)) : __popc((uint32_t)(kept & lt)));
            else
              to = start + (isp ? __popcll(kept) + __popcll(grp & pm & lt) : __popcll(kept & lt));
          }
          sg[r] = redc_mul(X.L[NP * MP + i], sig[r], M);
          dl = del[r] - (isp ? 1 : 0);  // src/sigma_basis.rs:408-411
        }
        // sigma by row; delta and the source row by position of the next order
        X.perm[to] = i;
        X.del[to] = dl;
        X.sig[i] = sg[r];
        if (leaf + 1 == K) {  // delta and the row scales of the block, in row order
          if (i < m) P.delta[i] = dbase + dl;
          for (int q = 1 + P.nres; q < csize; ++q)
            st_async(peer_addr(sm + S::OFF_SIG + i, q), sg[r], peer_addr(sm + 2 * K, q));
        }
      }
    }
    if (leaf + 1 == K) return;
    if (warp < S::PWARPS) leaf_products<RL, CPW, EW>(P, X, leaf, m - (int)X.mask[2]);
    __syncthreads();
  }
}

template <int RL, int CPW, int EW>
__device__ void leaf_cta(const LeafBlock& P, uint32_t* sm, volatile int* s_abort, volatile int* s_ok) {
  const LeafScratch<RL, CPW, EW> X(sm);
  const int m = P.m, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // stable sort of delta, descending (src/sigma_basis.rs:357-359); offsets
  // from delta[0] fit 32 bits
  if (warp == 0) {
    const int64_t dbase = P.delta[0];
    int del[RL];
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      const int i = lane + 32 * r;
      del[r] = i < m ? (int)(P.delta[i] - dbase) : 0;
      X.row[i] = del[r];
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      const int i = lane + 32 * r;
      int pos = i;
      if (i < m) {
        pos = 0;
        for (int j = 0; j < m; ++j) pos += (X.row[j] > del[r]) || (X.row[j] == del[r] && j < i);
      }
      X.perm[pos] = i;
      X.del[pos] = del[r];
      X.sig[i] = 1;
    }
  }
  __syncthreads();
  if (warp < EW) leaf_eliminate<RL, CPW, EW>(P, sm, s_ok);
  else leaf_help<RL, CPW, EW>(P, sm, s_abort, s_ok);
}

// ---------------------------------------------------------------- residual and basis CTAs
// Waits for transform `leaf`; then the whole CTA unpacks it into byte planes
// (the buffers alternate): row i holds L^{-1}[i][slot] at the slots' source rows and, without a
// pivot of its own, the diagonal at its own source row.
template <int RL, int CPW, int EW>
__device__ bool receive_transform(const LeafBlock& P, uint32_t* sm, int leaf, int rank, volatile int* s_abort,
                                  unsigned long long& mask) {
  using S = LeafShape<RL, CPW, EW>;
  constexpr int MP = S::MP, KW = S::KW;
  const bool ok = bar_wait(sm, leaf, s_abort, P);
  __syncwarp();
  const uint32_t* L = sm + S::OFF_RING + (leaf % S::slots(P.K)) * S::LW;
  uint32_t* Tp = sm + S::OFF_T + (leaf & 1) * S::TW;
  mask = L[S::MASK] | ((unsigned long long)L[S::MASK + 1] << 32);
  for (int e = ok ? threadIdx.x : MP * KW; e < MP * KW; e += kThreads) {
    const int i = e / KW, w = e % KW;
    const uint4 mp = *reinterpret_cast<const uint4*>(L + S::MAP + 4 * w);
    const uint32_t slot[4] = {mp.x >> 8, mp.y >> 8, mp.z >> 8, mp.w >> 8};
    const int own = (int)(L[S::MAP + i] & 255u);
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = slot[j] != 255u ? L[slot[j] * MP + i] : (own == 4 * w + j ? L[S::DIAG + i] : 0u);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t lo = __byte_perm(v[0], v[1], 0x40 + 0x11 * l) & 0xffffu;
      const uint32_t hi = __byte_perm(v[2], v[3], 0x40 + 0x11 * l) & 0xffffu;
      Tp[l * MP * KW + plane_word<RL>(i, w)] = lo | (hi << 16);
    }
  }
  if (!__syncthreads_and(ok)) return false;
  if (S::kRinged && threadIdx.x == 0)  // the ring slot is free
    st_peer_release(peer_addr(sm + S::OFF_USED + rank, 0), (uint32_t)leaf + 1);
  return true;
}

// The products of one leaf in a residual (BASIS = false) or basis CTA: every
// warp keeps one 16-row strip of T and one 8-column tile and walks the
// coefficients, the first two (coefficient 1 of the next residual comes from
// them) by the first two groups of warps.
template <int RL, int CPW, int EW, bool BASIS>
__device__ void update_cta(const LeafBlock& P, uint32_t* sm, int rank, volatile int* s_abort) {
  using S = LeafShape<RL, CPW, EW>;
  constexpr int PW = S::PW, CC = S::CC, NTC = S::NTC;
  const int m = P.m, n = P.n, K = P.K, MT = (m + 15) / 16;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int cbase = (rank - 1 - (BASIS ? P.nres : 0)) * CC;
  const ModP M = P.M;
  // 2^32 and 2^48 mod p, and 2^16 where the compiler does not see it
  const uint32_t Wt[3] = {M.c32, (uint32_t)((uint64_t)M.c32 * 65536 % M.p), P.two16};
  uint32_t* const V = sm + S::OFF_RING + S::slots(K) * S::LW;
  const int combos = MT * NTC, groups = kWarps / combos;
  const int nt = warp % NTC, mt = (warp / NTC) % MT, group = warp / combos;
  const bool work = group < groups;
  int byte[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) byte[v] = plane_byte<RL>(nt * 8 + 2 * t4 + (v & 1), mt * 16 + g + 8 * (v >> 1));
  const int leaves = BASIS ? K : K - 2;
  for (int leaf = 0; leaf < leaves; ++leaf) {
    unsigned long long mx;
    if (!receive_transform<RL, CPW, EW>(P, sm, leaf, rank, s_abort, mx)) return;
    if (!work) continue;
    const uint32_t* Vc = V + (size_t)(leaf & 1) * (K + 1) * PW;
    uint32_t* Vn = V + (size_t)((leaf + 1) & 1) * (K + 1) * PW;
    uint32_t A[RL][4][4];
    load_rows<RL>(sm + S::OFF_T + (leaf & 1) * S::TW, mt, g, t4, A);
    // this lane's row of the four byte matrices of a whole tile: limb lane / 8, column lane % 8
    const uint32_t tile = smem_addr(Vn + (lane >> 3) * (CC * S::KW) + plane_word<RL>(nt * 8 + (lane & 7), 4 * mt));
    const int x[2] = {(int)((mx >> (mt * 16 + g)) & 1ull), (int)((mx >> (mt * 16 + g + 8)) & 1ull)};
    // A tile's rows g and its rows g + 8 usually share x: then the tile is
    // stored whole, as four transposed byte matrices, or as two halves.
    const int x0 = __shfl_sync(0xffffffffu, x[0], 0), x1 = __shfl_sync(0xffffffffu, x[1], 0);
    const bool halves = __all_sync(0xffffffffu, x[0] == x0 && x[1] == x1), whole = halves && x0 == x1;
    const int rem = K - leaf - 1;              // residual: coefficients left, outputs t in [1, rem)
    const int lo = BASIS ? 0 : 1, hi = BASIS ? leaf + 2 : rem;  // outputs t in [lo, hi)
    const int tq_end = BASIS ? leaf + 1 : rem + 1;
    const uint32_t r1 = peer_addr(sm + S::OFF_R1 + ((leaf + 1) & 1) * S::R1W, 0);
    const uint32_t bar = peer_addr(sm + 2 * leaf, 0);
    // The strip of T is often zero in half of its source rows (a strip of pivot
    // rows only has the pivots' source rows, and m <= 16 has no other half):
    // mode 0 or 1 = all in that half, 2 = both.
    int mode = 2;
    uint32_t H[4][2], A1[1][4][4];
    if constexpr (RL == 1) {
      uint32_t h0 = 0, h1 = 0;
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        h0 |= A[0][l][0] | A[0][l][1];
        h1 |= A[0][l][2] | A[0][l][3];
      }
      if (!__any_sync(0xffffffffu, h1)) mode = 0;
      else if (!__any_sync(0xffffffffu, h0)) mode = 1;
#pragma unroll
      for (int l = 0; l < 4; ++l)
#pragma unroll
        for (int q = 0; q < 2; ++q) H[l][q] = mode == 1 ? A[0][l][2 + q] : A[0][l][q];
    } else {
      uint32_t h0 = 0, h1 = 0;
#pragma unroll
      for (int l = 0; l < 4; ++l)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          h0 |= A[0][l][q];
          h1 |= A[RL - 1][l][q];
        }
      if (!__any_sync(0xffffffffu, h1)) mode = 0;
      else if (!__any_sync(0xffffffffu, h0)) mode = 1;
#pragma unroll
      for (int l = 0; l < 4; ++l)
#pragma unroll
        for (int q = 0; q < 4; ++q) A1[0][l][q] = mode == 1 ? A[RL - 1][l][q] : A[0][l][q];
    }
    for (int tq = lo + group; tq < tq_end; tq += groups) {
      uint32_t val[4];
      const uint32_t* Vq = Vc + tq * PW;
      if (mode == 2) tile_product<RL, RL>(A, Vq, 0, nt, g, t4, Wt, M, val);
      else if constexpr (RL == 1) tile_product_half(H, Vq, 4 * mode, nt, g, t4, Wt, M, val);
      else tile_product<RL, 1>(A1, Vq, 8 * mode, nt, g, t4, Wt, M, val);
      const int tb = BASIS ? tq : tq - 1;      // coefficient of the rows with x = 0
      if (!BASIS && tq <= 2) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int row = mt * 16 + g + 8 * (v >> 1), c = cbase + nt * 8 + 2 * t4 + (v & 1);
          if (tb + x[v >> 1] == 1 && row < m && c < n)
            st_async(r1 + 4u * (uint32_t)(row * S::RS1 + c), val[v], bar);
        }
      }
      if (whole) {
        const int t = tb + x0;
        if (t >= lo && t < hi) {
          uint32_t w[4];
          byte_transpose4(val, w);
          stmatrix_u8(tile + 4u * (uint32_t)(t * PW), w);
        }
        if (BASIS && (x0 ? tq == 0 : tq == leaf)) {  // the end of the rows' range that no product reaches
          const uint32_t w[4] = {0, 0, 0, 0};
          stmatrix_u8(tile + 4u * (uint32_t)((x0 ? 0 : leaf + 1) * PW), w);
        }
      } else {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int xr = halves ? (v < 2 ? x0 : x1) : x[v >> 1];
          const int t = tb + xr;
          if (t >= lo && t < hi) plane_store<RL>(Vn + t * PW, byte[v], val[v]);
          if (BASIS && (xr ? tq == 0 : tq == leaf)) plane_store<RL>(Vn + (xr ? 0 : leaf + 1) * PW, byte[v], 0u);
        }
      }
    }
  }
  if (!BASIS) return;
  // normalise by the row scales
  const bool ok = bar_wait(sm, K, s_abort, P);
  __syncwarp();
  if (!__syncthreads_and(ok)) return;
  uint32_t* inv = sm + S::OFF_T;
  if (tid < m) inv[tid] = inverse_r(sm[S::OFF_SIG + tid], M);
  __syncthreads();
  const uint32_t* Vc = V + (size_t)(K & 1) * (K + 1) * PW;
  const int cols = min(CC, m - cbase);
  for (int e = tid; e < m * cols * (K + 1); e += kThreads) {
    const int t = e % (K + 1), q = e / (K + 1), j = q % cols, r = q / cols;
    P.Mout[(int64_t)r * P.out_rs + (int64_t)(cbase + j) * P.out_cs + t] =
        redc_mul(plane_load<RL>(Vc + t * PW, plane_byte<RL>(j, r)), inv[r], M);
  }
}

template <int RL, int CPW, int EW>
__global__ void __launch_bounds__(kThreads, 1) pm_leaf_block_kernel(LeafBlock P) {
  using S = LeafShape<RL, CPW, EW>;
  extern __shared__ __align__(16) uint32_t leaf_smem[];
  __shared__ int s_abort, s_ok;
  uint32_t* const sm = leaf_smem;
  const int tid = threadIdx.x;
  const int csize = 1 + P.nres + P.nbas;
  const int rank = (int)(blockIdx.x % csize);  // clusters are consecutive blocks
  const int z = (int)(blockIdx.x / csize);
  P.G += (int64_t)z * P.g_bs;
  P.delta += (int64_t)z * P.m;
  P.Mout += (int64_t)z * P.out_bs;
  const int m = P.m, n = P.n, K = P.K;
  if (tid == 0) {
    s_abort = 0;
    s_ok = 1;
  }
  if (tid < 8) sm[S::OFF_USED + tid] = 0;
  // one mbarrier per message: transforms (and the row scales) in, coefficient 1 back
  if (tid <= K)
    bar_arm(sm, tid, (rank != 0 && tid == 0 ? 4u * (uint32_t)P.missing : 0u) + (rank == 0 ? (uint32_t)(4 * m * n) : tid == K ? 4u * S::MP : (uint32_t)(4 * ((n + 2) * S::MP + 2))));
  if (rank == 0) {
    for (int e = S::OFF_R1 + tid; e < S::OFF_FB; e += kThreads) sm[e] = 0;
    __syncthreads();
    for (int e = tid; e < m * n; e += kThreads) {  // coefficients 0 and 1
      const uint32_t* src = P.G + (int64_t)(e / n) * P.g_rs + (int64_t)(e % n) * P.g_cs;
      sm[S::OFF_R0 + (e / n) * S::RS0 + e % n] = src[0];
      if (K > 1) sm[S::OFF_R1 + (e / n) * S::RS1 + e % n] = src[1];
    }
  } else {
    uint32_t* V = sm + S::OFF_RING + S::slots(K) * S::LW;
    for (int e = tid; e < 2 * (K + 1) * S::PW; e += kThreads) V[e] = 0;
    __syncthreads();
    if (rank <= P.nres) {
      // a warp per entry (i, c), a lane per coefficient, eight entries in flight
      const int cbase = (rank - 1) * S::CC, cols = min(S::CC, n - cbase), lane = tid & 31;
      for (int t = lane; t - lane < K; t += 32)
        for (int q0 = tid >> 5; q0 < m * cols; q0 += 8 * kWarps) {
          uint32_t v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int q = q0 + u * kWarps, i = q / cols, c = q - i * cols;
            v[u] = q < m * cols && t < K ? P.G[(int64_t)i * P.g_rs + (int64_t)(cbase + c) * P.g_cs + t] : 0u;
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int q = q0 + u * kWarps, i = q / cols, c = q - i * cols;
            if (q < m * cols && t < K) plane_store<RL>(V + t * S::PW, plane_byte<RL>(c, i), v[u]);
          }
        }
    } else if (tid < S::CC) {
      const int j = (rank - 1 - P.nres) * S::CC + tid;
      if (j < m) plane_store<RL>(V, plane_byte<RL>(tid, j), 1u);  // V_0 = identity
    }
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  cluster_sync();
  if (rank == 0) {
    leaf_cta<RL, CPW, EW>(P, sm, &s_abort, &s_ok);
  } else if (rank <= P.nres) {
    update_cta<RL, CPW, EW, false>(P, sm, rank, &s_abort);
  } else {
    update_cta<RL, CPW, EW, true>(P, sm, rank, &s_abort);
  }
  __syncwarp();
  // No CTA leaves while another may still write into its shared memory.  Every
  // message has been waited for, unless a wait of this CTA gave up: then those
  // still in flight, which all have been sent by now, get time to land.
  cluster_sync();
  if (*(volatile int*)&s_abort) {
    const uint64_t t0 = now_ns();
    while (now_ns() - t0 < kLandNs) __nanosleep(1000);
  }
}

template <int RL, int CPW, int EW>
int launch(LeafBlock P, int nb, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  const int csize = 1 + P.nres + P.nbas;
  cfg.gridDim = dim3((unsigned)(nb * csize));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = LeafShape<RL, CPW, EW>::smem_bytes(P.K);
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  P.two16 = 65536;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RR_CUDA(cudaLaunchKernelEx(&cfg, pm_leaf_block_kernel<RL, CPW, EW>, P));
  return RR_OK;
}

template <int RL, int CPW, int EW>
int set_limit(int K) {
  // always the largest size this variant launches: the limit is per kernel,
  // shared by every thread of the process
  static_assert(LeafShape<RL, CPW, EW>::smem_bytes(RL > 1 ? 16 : CPW <= 2 ? 64 : 32) <= 227 * 1024 - 1024, "shared memory");
  RR_CUDA(cudaFuncSetAttribute(pm_leaf_block_kernel<RL, CPW, EW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)LeafShape<RL, CPW, EW>::smem_bytes(K)));
  return RR_OK;
}

}  // namespace

// Leaves per block.  A leaf's residual and basis updates take one product per
// remaining (or finished) coefficient, spread over the cluster; at these sizes
// they stay near the time of an elimination, and the planes fit shared memory.
int leaf_block_max(int m) { return m <= 16 ? 64 : m <= 32 ? 32 : 16; }

int leaf_block_prepare(int n) {
  if (n <= 4) return set_limit<1, 1, 4>(64);
  if (n <= 8) return set_limit<1, 2, 4>(64);
  if (n <= 16) return set_limit<1, 4, 4>(32);
  return set_limit<2, 4, 8>(16);
}

int leaf_block_launch(LeafBlock P, int nb, cudaStream_t s) {
  const int cc = P.n <= 16 ? 8 : 16;
  P.nres = (P.n + cc - 1) / cc;
  P.nbas = (P.m + cc - 1) / cc;
  if (1 + P.nres + P.nbas > kMaxCluster || P.K > leaf_block_max(P.m))
    return fail(RR_EINVAL, "internal: leaf block m = %d, n = %d, K = %d", P.m, P.n, P.K);
  if (P.n <= 4) return launch<1, 1, 4>(P, nb, s);
  if (P.n <= 8) return launch<1, 2, 4>(P, nb, s);
  if (P.n <= 16) return launch<1, 4, 4>(P, nb, s);
  return launch<2, 4, 8>(P, nb, s);
}

}  // namespace rr
