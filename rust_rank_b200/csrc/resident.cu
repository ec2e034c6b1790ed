// resident.cu -- runs of applications of B on matrices that fit the chip: one
// launch per run, the CSR of A and of A^T in shared memory.
//
// Algebra and block layout as in krylov.cu; the run replaces its pass kernels
// where those are bound by latency: a pass over a 20,000-row matrix moves 2 MB
// and took 10 us, in launch, dependent loads (offsets, entries, gathers) and
// the finish of the Gram term, which the next pass waited for.  Here
//
//   * every CTA keeps the entries of its rows in shared memory for the whole
//     run (row batches of equal degree, padded to the longest row, so that an
//     entry is one conflict-free read);
//   * a pass is the gathers (from L2: the blocks are rewritten by other SMs),
//     the row epilogue and one grid barrier;
//   * a CTA's Gram warps read the rows it has just written and add their Gram
//     term while the other warps run the next pass; terms go to a slot each and
//     are reduced mod p once, after the run.
//
// Measured (us per application, B200; before: the pass kernels in a CUDA
// graph): 1500 x 1200, b = 4: 5.7 against 14.1; 20,000^2, b = 8: 7.2 against
// 21; 30,011 x 23,017, b = 5: 8.1 against 22; 194,003 x 151,007, b = 16:
// 45 against 63.  The small ones are bound by the barrier and one gather's
// latency; the last by the rate at which L2 serves random 64-byte rows
// (8500 gathers per SM and pass, 4.2 TB/s in all).
//
// The grid barrier gives up after a limit (2 s by default) of %globaltimer and
// sets *status; the CTA's other warps learn of it at their next CTA barrier.
#include <algorithm>
#include <mutex>

#include "krylov_gram.cuh"

namespace rr {

namespace {

constexpr int kGatherWarps = 16;
// Gram warps: at width 16 four of them take longer than a pass of the largest
// matrices that fit.
template <int B>
constexpr int kGramWarps = B >= 16 ? 8 : 4;
template <int B>
constexpr int kResThreads = 32 * (kGatherWarps + kGramWarps<B>);
constexpr int kMaxBatches = 512;  // row batches of one CTA, per matrix
constexpr int64_t kResMaxDegree = 64;
constexpr size_t kResSmem = 227 * 1024 - 2048;

struct ResCsr {
  const uint32_t* rowptr;
  const uint2* cv;
  int64_t rows;
};

struct ResParams {
  ResCsr A, At;
  uint4* X[2];
  uint4* U;
  int cur0;
  int apps;
  const uint32_t *dr_m, *dc_m, *dc_r, *drinv_r, *dcinv_r;
  unsigned long long* gram;  // [2 apps][NP], zero at launch
  unsigned int* bar;         // arrivals, zero at launch
  int* status;
  uint64_t limit_ns;         // a barrier wait gives up after this long
  unsigned int missing;      // arrivals the barriers expect beyond those that come (0; checks of the give-up path)
  ModP M;
  uint32_t w4, w5, w6;
};

__device__ __forceinline__ void gather_bar() { __barrier_sync_count(1, 32 * kGatherWarps); }
template <int B>
__device__ __forceinline__ void gram_bar() {
  __barrier_sync_count(2, 32 * kGramWarps<B>);
}

// The entries of a CTA's row batches (batch j of the CTA = batch blockIdx.x +
// j gridDim.x of the matrix), batch after batch, [step][slot] with zero entries
// past a row's end.  first[j] = the batch's first entry, first[count] = the end.
template <int B>
__device__ int load_entries(const ResCsr& C, uint2* ell, int* first) {
  constexpr int RPW = 128 / B;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t nbatch = (C.rows + RPW - 1) / RPW;
  const int count = blockIdx.x < nbatch ? (int)((nbatch - 1 - blockIdx.x) / gridDim.x) + 1 : 0;
  // rows are in decreasing degree order: the first row of a batch is its longest
  for (int j = tid; j < count; j += kResThreads<B>) {
    const int64_t r = ((int64_t)blockIdx.x + (int64_t)j * gridDim.x) * RPW;
    first[j + 1] = (int)(C.rowptr[r + 1] - C.rowptr[r]) * RPW;
  }
  __syncthreads();
  if (warp == 0) {
    int base = 0;
    for (int j0 = 0; j0 < count; j0 += 32) {
      int v = j0 + lane < count ? first[j0 + lane + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      if (j0 + lane < count) first[j0 + lane + 1] = base + v;
      base += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) first[0] = 0;
  }
  __syncthreads();
  for (int j = warp; j < count; j += kResThreads<B> / 32) {
    const int64_t r0 = ((int64_t)blockIdx.x + (int64_t)j * gridDim.x) * RPW;
    const int b0 = first[j], len = first[j + 1] - b0;
    for (int e = lane; e < len; e += 32) {
      const int64_t r = r0 + e % RPW;
      uint2 v = make_uint2(0u, 0u);
      if (r < C.rows) {
        const uint32_t k = C.rowptr[r] + (uint32_t)(e / RPW);
        if (k < C.rowptr[r + 1]) v = C.cv[k];
      }
      ell[b0 + e] = v;
    }
  }
  return count;
}

// acc += val * g for the four lanes of each of the first `n` loaded entries
template <int N>
__device__ __forceinline__ void mac_entries(const uint2 (&e)[N], const uint4 (&g)[N], const ModP& M, uint64_t (&acc)[4]) {
#pragma unroll
  for (int u = 0; u < N; ++u) {
    acc[0] += (uint64_t)e[u].y * g[u].x;
    acc[1] += (uint64_t)e[u].y * g[u].y;
    acc[2] += (uint64_t)e[u].y * g[u].z;
    acc[3] += (uint64_t)e[u].y * g[u].w;
    if ((u & 3) == 3) {  // four products fit between folds for every p < 2^31
#pragma unroll
      for (int l = 0; l < 4; ++l) acc[l] = fold(acc[l], M);
    }
  }
}

// One pass of the gather warps over the CTA's row batches: Y = scaled rows of C X.
template <int B, bool EVEN>
__device__ __forceinline__ void res_pass(const ResCsr& C, const uint2* ell, const int* first, int count, const uint4* X,
                                         uint4* Y, const uint32_t* __restrict__ scale,
                                         const uint32_t* __restrict__ scale2, const ModP& M) {
  constexpr int TPR = B / 4, RPW = 32 / TPR;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % TPR, slot = lane / TPR;
  const uint4* Xs = X + sub;
  for (int j = warp; j < count; j += kGatherWarps) {
    const int64_t r = ((int64_t)blockIdx.x + (int64_t)j * gridDim.x) * RPW + slot;
    const bool on = r < C.rows;
    const uint32_t s1 = on ? __ldg(scale + r) : 0u;
    const uint32_t s2 = EVEN && on ? __ldg(scale2 + r) : 0u;
    const uint2* ep = ell + first[j] + slot;
    int left = (first[j + 1] - first[j]) / RPW;
    uint64_t acc[4] = {0, 0, 0, 0};
    for (; left >= 8; left -= 8, ep += 8 * RPW) {
      uint2 e[8];
      uint4 g[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) e[u] = ep[u * RPW];
#pragma unroll
      for (int u = 0; u < 8; ++u) g[u] = __ldcg(Xs + (size_t)e[u].x * TPR);
      mac_entries<8>(e, g, M, acc);
    }
    if (left > 0) {  // the same count in every lane
      uint2 e[7];
      uint4 g[7];
#pragma unroll
      for (int u = 0; u < 7; ++u) e[u] = u < left ? ep[u * RPW] : make_uint2(0u, 0u);
#pragma unroll
      for (int u = 0; u < 7; ++u) {
        g[u] = make_uint4(0, 0, 0, 0);
        if (u < left) g[u] = __ldcg(Xs + (size_t)e[u].x * TPR);
      }
      mac_entries<7>(e, g, M, acc);
    }
    if (on) {
      uint32_t o[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        o[l] = redc((uint64_t)redc(fold(acc[l], M), M) * s1, M);  // d_r z, or w'
        if (EVEN) o[l] = redc((uint64_t)o[l] * s2, M);              // d_c w'
      }
      __stcg(Y + r * TPR + sub, make_uint4(o[0], o[1], o[2], o[3]));
    }
  }
}

// The Gram term of the CTA's rows of Y: odd z (x) Y with z = Y d_r^{-1}, even
// w (x) w with w = Y d_c^{-1}.  Four batches are loaded before the first is used.
template <int B, bool EVEN, class Gram>
__device__ __forceinline__ void res_gram(Gram& gram, int64_t rows, int count, const uint4* Y,
                                         const uint32_t* __restrict__ inv, const ModP& M, const uint32_t (&W)[3],
                                         uint32_t* part, unsigned long long* out) {
  constexpr int TPR = B / 4, RPW = 32 / TPR;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) - kGatherWarps, sub = lane % TPR, slot = lane / TPR;
  for (int j0 = warp; j0 < count; j0 += 4 * kGramWarps<B>) {
    uint4 y[4];
    uint32_t s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u * kGramWarps<B>;
      const int64_t r = ((int64_t)blockIdx.x + (int64_t)j * gridDim.x) * RPW + slot;
      const bool on = j < count && r < rows;
      y[u] = on ? __ldcg(Y + r * TPR + sub) : make_uint4(0, 0, 0, 0);
      s[u] = on ? __ldg(inv + r) : 0u;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j0 + u * kGramWarps<B> >= count) break;
      const uint32_t v[4] = {y[u].x, y[u].y, y[u].z, y[u].w};
      uint32_t z[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) z[l] = redc((uint64_t)v[l] * s[u], M);
      if (EVEN) gram.add_sym(z, slot, sub, lane, M, W);
      else gram.add(z, v, slot, sub, lane, M, W);
    }
  }
  if (EVEN) gram.finish_sym(slot, sub, lane, M, W);
  else gram.finish(slot, sub, lane, M, W);
  gram.store(part + warp * B * B, lane, M);
  gram.reset();
  gram_bar<B>();
  for (int e = threadIdx.x - 32 * kGatherWarps; e < B * B; e += 32 * kGramWarps<B>) {
    const int i = e / B, c = e % B;
    if (i <= c) {
      unsigned long long v = 0;
#pragma unroll
      for (int w = 0; w < kGramWarps<B>; ++w) v += part[w * B * B + e];
      if (v) atomicAdd(out + pair_index(i, c, B), v);
    }
  }
  gram_bar<B>();
}

template <int B>
using ResGram = typename std::conditional<(B >= 8), GramMma<B, 4>, GramCore<B, 4>>::type;

template <int B>
constexpr size_t res_fixed_smem() {  // Gram staging, the Gram warps' sums, batch offsets
  return (size_t)4 * kGramWarps<B> * (ResGram<B>::kWords + B * B) + 4 * 2 * (kMaxBatches + 2);
}

template <int B>
__global__ void __launch_bounds__(kResThreads<B>, 1) resident_kernel(ResParams P, int entriesA) {
  constexpr int NP = B * (B + 1) / 2;
  extern __shared__ __align__(16) unsigned char res_smem[];
  // s_stop[p & 1]: the run ends at the CTA barrier of pass p.  Thread 0 sets it
  // after the barrier of pass p - 1, when a Gram warp may still have to read the
  // flag of p - 1: with one flag for both, some of the Gram warps could leave and
  // the others wait for them in gram_bar.
  __shared__ volatile int s_stop[2];
  uint2* const ellA = reinterpret_cast<uint2*>(res_smem + res_fixed_smem<B>());
  uint2* const ellAt = ellA + entriesA;
  uint32_t* const staging = reinterpret_cast<uint32_t*>(res_smem);
  uint32_t* const part = staging + (size_t)kGramWarps<B> * ResGram<B>::kWords;
  int* const firstA = reinterpret_cast<int*>(part + kGramWarps<B> * B * B);
  int* const firstAt = firstA + kMaxBatches + 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const ModP M = P.M;
  if (tid < 2) s_stop[tid] = 0;
  const int nA = load_entries<B>(P.A, ellA, firstA);
  const int nAt = load_entries<B>(P.At, ellAt, firstAt);
  __syncthreads();
  if (warp < kGatherWarps) {
    int cur = P.cur0;
    unsigned int target = P.missing;
    for (int p = 0; p < 2 * P.apps; ++p) {
      if ((p & 1) == 0) {
        res_pass<B, false>(P.A, ellA, firstA, nA, P.X[cur], P.U, P.dr_m, nullptr, M);
      } else {
        res_pass<B, true>(P.At, ellAt, firstAt, nAt, P.U, P.X[cur ^ 1], P.dc_m, P.dc_r, M);
        cur ^= 1;
      }
      __syncthreads();  // the rows are written, and the Gram warps are done with the previous pass
      if (p + 1 == 2 * P.apps) break;
      target += gridDim.x;
      if (tid == 0) {
        // one arrival per CTA; all CTAs wait on the same word (a release word of
        // its own, written by the last to arrive, was 2 us slower per application)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.bar) : "memory");
        uint64_t t0 = 0;
        for (int spins = 0;; ++spins) {
          unsigned int seen;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(P.bar) : "memory");
          if (seen >= target) break;
          if ((spins & 255) == 255) {
            const uint64_t t = now_ns();
            if (t0 == 0) t0 = t;
            if (*(volatile int*)P.status || t - t0 > P.limit_ns) {
              atomicExch(P.status, 1);
              s_stop[(p + 1) & 1] = 1;
              break;
            }
          }
        }
      }
      gather_bar();
      if (s_stop[(p + 1) & 1]) {
        __syncthreads();  // the barrier of pass p + 1, after which the Gram warps leave too
        break;
      }
    }
  } else {
    ResGram<B> gram;
    gram.init(staging + (size_t)(warp - kGatherWarps) * ResGram<B>::kWords, lane);
    const uint32_t W[3] = {P.w4, P.w5, P.w6};
    int cur = P.cur0;
    for (int p = 0; p < 2 * P.apps; ++p) {
      __syncthreads();
      if (s_stop[p & 1]) break;
      unsigned long long* out = P.gram + (size_t)p * NP;
      if ((p & 1) == 0) {
        res_gram<B, false>(gram, P.A.rows, nA, P.U, P.drinv_r, M, W, part, out);
      } else {
        res_gram<B, true>(gram, P.At.rows, nAt, P.X[cur ^ 1], P.dcinv_r, M, W, part, out);
        cur ^= 1;
      }
    }
  }
}

// Cooperative grids of one device.  Grids that together need more SMs than
// there are must not be in flight together: each could hold some SMs and wait
// for the rest.  So a run takes a share of the device, 1 / 2^level of its SMs
// (slot j of level l is [j, j + 1) sms / 2^l), and waits, through events, for
// the last runs of the parts it takes; two runs in flight never share a part,
// and waits only go back to runs queued earlier.  None is queued while a batch
// holds the device.
//
// Level: a run alone on the device takes all the SMs it has row batches for;
// when the streams of k other contexts have runs in flight, 1 / (k + 1) of
// them, as far down as the matrix still fits the share's shared memory.  These
// runs are bound by latency, so side by side they lose little each.  Measured
// (ms for 256 applications in each of 8 contexts; pass kernels / runs of the
// whole device one after the other / side by side): 700 rows, b = 4: 4.1 / 11.2 /
// 2.2; 5000 rows, b = 8: 5.5 / 14.0 / 3.7; 20,000 rows, b = 8: 8.2 / 15.7 / 7.8;
// 64 applications, 60,000 rows, b = 16: 14.8 / 10.1 / 8.8.
//
// Runs of fewer than kResShort applications (width 16 only, see queue_apps) are
// taken alone on the device only: among others the pass kernels are as good or
// better (8 contexts, 64 applications of 2000 rows one by one: 6.0 ms with runs,
// 5.2 without; 32 of 20,000 rows: 3.4 / 3.2).
constexpr int kResShort = 4;
constexpr int kCoopLevels = 4;               // the smallest share: 1/16, 9 SMs
constexpr int kCoopParts = 1 << kCoopLevels;

struct CoopChain {
  struct Run {
    cudaEvent_t done = nullptr;
    cudaStream_t stream = nullptr;
    uint64_t seq = 0;        // order of queuing
    int parts = 0;           // parts whose last run this is; 0 = a free record
    bool finished = false;   // seen complete
  };
  std::mutex m;
  Run runs[kCoopParts + 1];  // as many as can be the last run of a part, and one to fill in
  Run* last[kCoopParts] = {};
  uint64_t seq = 0;
  int holds = 0;             // batches with persistent launches in flight

  bool pending(const Run& r, cudaStream_t s) const { return r.parts > 0 && !r.finished && r.stream != s; }
  // stream s waits for run r
  int wait(cudaStream_t s, const Run& r) {
    if (pending(r, s)) RR_CUDA(cudaStreamWaitEvent(s, r.done, 0));
    return RR_OK;
  }
  // Streams other than s with runs in flight.
  int others(cudaStream_t s) {
    int n = 0;
    // an event query is not allowed while any thread captures in the global mode
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    bool asked = false;
    for (Run& r : runs) {
      if (!pending(r, s)) continue;
      if (!asked) cudaThreadExchangeStreamCaptureMode(&mode);
      asked = true;
      const cudaError_t e = cudaEventQuery(r.done);
      r.finished = e == cudaSuccess;
      if (r.finished) continue;
      cudaGetLastError();  // not ready is not an error
      bool seen = false;
      for (const Run* q = runs; q != &r && !seen; ++q) seen = pending(*q, s) && q->stream == r.stream;
      n += !seen;
    }
    if (asked) cudaThreadExchangeStreamCaptureMode(&mode);
    return n;
  }
};
constexpr int kMaxDevices = 64;
CoopChain g_coop[kMaxDevices];

// A run's turn: its level and the wait for the parts it takes, held until the
// run is queued.
class CoopTurn {
 public:
  // The run may go from level `top` (it has no use for more SMs) to `deepest`
  // (it does not fit fewer); *level = the one it takes, -1 = none: a batch holds
  // the device, or (alone_only) other streams have runs in flight.
  int begin(int device, cudaStream_t s, int top, int deepest, bool alone_only, int* level) {
    *level = -1;
    if (device < 0 || device >= kMaxDevices) return RR_OK;
    c_ = &g_coop[device];
    c_->m.lock();
    if (c_->holds > 0) return RR_OK;
    const int streams = c_->others(s) + 1;
    if (alone_only && streams > 1) return RR_OK;
    int l = top;
    while ((1 << l) < streams && l < deepest) ++l;
    const int width = kCoopParts >> l;
    // the slot whose runs of other streams were queued the longest ago, or that has none
    uint64_t best = ~0ull;
    for (int j = 0; j < kCoopParts; j += width) {
      uint64_t newest = 0;
      for (int q = j; q < j + width; ++q)
        if (c_->last[q] && c_->pending(*c_->last[q], s)) newest = std::max(newest, c_->last[q]->seq);
      if (newest < best) {
        best = newest;
        first_ = j;
      }
    }
    width_ = width;
    for (int q = first_; q < first_ + width; ++q)
      if (c_->last[q] && (q == first_ || c_->last[q] != c_->last[q - 1])) RR_TRY(c_->wait(s, *c_->last[q]));
    stream_ = s;
    *level = l;
    return RR_OK;
  }
  // The run is queued.
  int end() {
    CoopChain::Run* r = c_->runs;
    while (r->parts > 0) ++r;
    cudaError_t e = r->done ? cudaSuccess : cudaEventCreateWithFlags(&r->done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(r->done, stream_);
    if (e != cudaSuccess) {  // nobody could wait for the run
      cudaStreamSynchronize(stream_);
      RR_CUDA(e);
    }
    for (int q = first_; q < first_ + width_; ++q) {
      if (c_->last[q]) --c_->last[q]->parts;
      c_->last[q] = r;
    }
    r->stream = stream_;
    r->seq = ++c_->seq;
    r->parts = width_;
    r->finished = false;
    return RR_OK;
  }
  ~CoopTurn() {
    if (c_) c_->m.unlock();
  }

 private:
  CoopChain* c_ = nullptr;
  cudaStream_t stream_ = nullptr;
  int first_ = 0, width_ = 0;
};

// Gram sums of `terms` terms -> sequence terms (real pairs); the sums, the
// barrier and the device term counter are made ready for the next launch.
__global__ void resident_finish_kernel(unsigned long long* gram, int terms, int b, int B, uint32_t* S,
                                       unsigned int* term_ctr, unsigned int* bar, ModP M) {
  const int NP = B * (B + 1) / 2, npr = b * (b + 1) / 2;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < terms * NP; e += gridDim.x * blockDim.x) {
    const int t = e / NP;
    int i, j;
    pair_of(e - t * NP, B, i, j);
    if (j < b) S[(size_t)t * npr + pair_index(i, j, b)] = reduce(gram[e], M);
    gram[e] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *term_ctr += (unsigned)terms;
    *bar = 0;
  }
}

// Entries of a CTA for one matrix, at most: the row batches of a CTA are every
// grid-th one of a list of non-increasing lengths, so all but its first are
// bounded by the mean of the lengths before them.
int64_t entry_bound(int64_t nnz, int64_t max_degree, int rpw, int grid) {
  return rpw * max_degree + (nnz + rpw * max_degree) / grid + 1;
}

// The grid of a matrix at a level, its entries of A per CTA and its dynamic
// shared memory (0 = it does not fit).
struct ResShape {
  int grid, entriesA;
  size_t smem;
};
template <int B>
ResShape shape_at(const rr_matrix* mat, int level) {
  constexpr int RPW = 128 / B;
  const int64_t batches = (std::max(mat->m, mat->n) + RPW - 1) / RPW;
  ResShape r{(int)std::min<int64_t>(batches, mat->ctx->num_sms >> level), 0, 0};
  if (r.grid == 0 || (batches + r.grid - 1) / r.grid > kMaxBatches) return r;
  const int64_t ea = entry_bound(mat->nnz, mat->max_row_nnz, RPW, r.grid);
  const size_t smem = res_fixed_smem<B>() + 8 * (size_t)(ea + entry_bound(mat->nnz, mat->max_col_nnz, RPW, r.grid));
  if (smem > kResSmem) return r;
  r.entriesA = (int)ea;
  r.smem = smem;
  return r;
}

template <int B>
int prepare(rr_krylov* kr) {
  constexpr int RPW = 128 / B;
  const rr_matrix* mat = kr->mat;
  kr->res_deepest = -1;
  if (mat->max_row_nnz > kResMaxDegree || mat->max_col_nnz > kResMaxDegree) return RR_OK;
  for (int l = 0; l <= kCoopLevels && shape_at<B>(mat, l).smem > 0; ++l) kr->res_deepest = l;
  if (kr->res_deepest < 0) return RR_OK;
  const int64_t batches = (std::max(mat->m, mat->n) + RPW - 1) / RPW;
  kr->res_top = 0;
  while (kr->res_top < kr->res_deepest && (mat->ctx->num_sms >> (kr->res_top + 1)) >= batches) ++kr->res_top;
  if (mat->ctx->coop_level <= kr->res_deepest) kr->res_top = std::max(kr->res_top, mat->ctx->coop_level);
  kr->res_apps = std::min(mat->ctx->run_apps, kResMaxApps);
  return RR_OK;
}

// At a handle's first run: its Gram slots, and behind them the barrier word.
// Without room for them the handle takes the pass kernels.
template <int B>
int scratch(rr_krylov* kr) {
  // the limit is per kernel, shared by every thread of the process: always the largest
  RR_CUDA(cudaFuncSetAttribute(resident_kernel<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem));
  cudaStream_t s = kr->mat->ctx->stream;
  if (kr->res_gram.alloc_async(resident_gram_words(B, kr->res_apps) + 1, s) != RR_OK) {
    kr->res_deepest = -1;
    return RR_OK;
  }
  RR_CUDA(cudaMemsetAsync(kr->res_gram.ptr, 0, kr->res_gram.bytes(), s));
  kr->res_bar = reinterpret_cast<unsigned int*>(kr->res_gram.ptr + resident_gram_words(B, kr->res_apps));
  return RR_OK;
}

template <int B>
int run(rr_krylov* kr, int apps, bool* taken) {
  const rr_matrix* mat = kr->mat;
  cudaStream_t s = mat->ctx->stream;
  *taken = false;
  if (!kr->res_bar) RR_TRY(scratch<B>(kr));
  if (!kr->res_bar) return RR_OK;
  ResParams P;
  P.A = ResCsr{mat->A.rowptr.ptr, mat->A.cv.ptr, mat->A.rows};
  P.At = ResCsr{mat->At.rowptr.ptr, mat->At.cv.ptr, mat->At.rows};
  P.X[0] = reinterpret_cast<uint4*>(kr->X[0].ptr);
  P.X[1] = reinterpret_cast<uint4*>(kr->X[1].ptr);
  P.U = reinterpret_cast<uint4*>(kr->U.ptr);
  P.cur0 = kr->cur;
  P.apps = apps;
  P.dr_m = kr->dr_m.ptr;
  P.dc_m = kr->dc_m.ptr;
  P.dc_r = kr->dc_r.ptr;
  P.drinv_r = kr->drinv_r.ptr;
  P.dcinv_r = kr->dcinv_r.ptr;
  P.gram = kr->res_gram.ptr;
  P.bar = kr->res_bar;
  P.status = kr->d_status.ptr;
  P.limit_ns = mat->ctx->wait_limit_ns;
  P.missing = (unsigned int)mat->ctx->wait_missing;
  P.M = kr->M;
  P.w4 = kr->M.c32;
  P.w5 = (uint32_t)((uint64_t)P.w4 * 256 % kr->M.p);
  P.w6 = (uint32_t)((uint64_t)P.w5 * 256 % kr->M.p);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.blockDim = dim3(kResThreads<B>);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  {
    CoopTurn turn;
    int level;
    RR_TRY(turn.begin(mat->ctx->device, s, kr->res_top, kr->res_deepest, apps < kResShort, &level));
    *taken = level >= 0;
    if (!*taken) return RR_OK;
    const ResShape shape = shape_at<B>(mat, level);
    cfg.gridDim = dim3((unsigned)shape.grid);
    cfg.dynamicSmemBytes = shape.smem;
    RR_CUDA(cudaLaunchKernelEx(&cfg, resident_kernel<B>, P, shape.entriesA));
    RR_TRY(turn.end());
  }
  const int np = kr->b * (kr->b + 1) / 2, NP = B * (B + 1) / 2;
  resident_finish_kernel<<<std::min((2 * apps * NP + 255) / 256, 296), 256, 0, s>>>(
      kr->res_gram.ptr, 2 * apps, kr->b, B, kr->S.ptr + (size_t)(kr->len - kr->base) * np, kr->d_term.ptr,
      kr->res_bar, kr->M);
  RR_CUDA(cudaGetLastError());
  kr->launches += 2;
  kr->len += 2 * apps;
  kr->cur ^= apps & 1;
  return RR_OK;
}

}  // namespace

int CoopHold::begin(int device, cudaStream_t s) {
  if (device < 0 || device >= kMaxDevices) return RR_OK;
  CoopChain& c = g_coop[device];
  std::lock_guard<std::mutex> lk(c.m);
  for (const CoopChain::Run& r : c.runs) RR_TRY(c.wait(s, r));
  device_ = device;
  ++c.holds;
  return RR_OK;
}

CoopHold::~CoopHold() {
  if (device_ < 0) return;
  std::lock_guard<std::mutex> lk(g_coop[device_].m);
  --g_coop[device_].holds;
}

int resident_prepare(rr_krylov* kr) {
  switch (kr->B) {
    case 4: return prepare<4>(kr);
    case 8: return prepare<8>(kr);
    case 16: return prepare<16>(kr);
  }
  kr->res_deepest = -1;
  return RR_OK;
}

int resident_run(rr_krylov* kr, int apps, bool* taken) {
  switch (kr->B) {
    case 4: return run<4>(kr, apps, taken);
    case 8: return run<8>(kr, apps, taken);
    case 16: return run<16>(kr, apps, taken);
  }
  return fail(RR_EINVAL, "no resident run at width %d", kr->B);
}

}  // namespace rr
