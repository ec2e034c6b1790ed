// upload.cpp -- copies between the caller's host arrays and the device.
//
// Matrices and blocks arrive as ordinary (pageable) host memory: numpy arrays,
// Rust Vecs.  A cudaMemcpyAsync from pageable memory is staged by the driver
// through its own pinned buffer on the calling thread alone.  Here several host
// threads copy pieces into pinned staging buffers of the context while the
// pieces copied before them are in flight over the bus: the host copies and
// the transfers overlap, and the host copy itself runs on several cores.
// Arrays already in pinned memory go straight to cudaMemcpyAsync.  Results leave
// the device the same way: a 96 MB block took 21 ms as one pageable copy (which
// also touches the fresh pages of the caller's array on one thread), 5 ms through
// the staging buffers.  Below 8 MB that pays only where the array's pages are
// still to be touched: into touched ones the driver's copy takes 0.29 ms for
// 4.5 MB and 0.36 for 6, the staged one anything from 0.29 to 0.66 (its threads'
// start is most of it); into fresh ones 2.5 and 3.3 ms against 1.5 and 1.9.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "rr_internal.h"

namespace rr {

namespace {
constexpr size_t kPiece = 2u << 20;     // bytes per staged piece
constexpr size_t kStageMin = 4u << 20;  // smaller copies go straight to the driver
constexpr size_t kStageTouched = 8u << 20;  // downloads into touched pages: staged from here on
constexpr int kMaxStageThreads = 8;
constexpr size_t kStageNew = 32u << 20;  // downloads a context creates its buffers for
}  // namespace

// Per-context staging: two pinned buffers and two events per copy thread,
// allocated at the first staged copy, freed with the context.
struct Staging {
  std::mutex mu;
  int threads = 0;
  std::vector<void*> buf;
  std::vector<cudaEvent_t> ev;
  ~Staging() {
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
    for (void* b : buf)
      if (b) cudaFreeHost(b);
  }
};

void staging_destroy(Staging* st) { delete st; }

static bool is_pinned(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

namespace {

// Whether at least half of the pages of [p, p + bytes) are there already (bytes
// below kStageTouched).
bool touched(const void* p, size_t bytes) {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  unsigned char there[kStageTouched / 4096 + 2];
  const uintptr_t lo = (uintptr_t)p / page * page, hi = (uintptr_t)p + bytes;
  const size_t n = (hi - lo + page - 1) / page;
  if (n > sizeof(there) || mincore((void*)lo, hi - lo, there) != 0) return false;
  size_t count = 0;
  for (size_t i = 0; i < n; ++i) count += there[i] & 1;
  return 2 * count >= n;
}

struct Piece {
  char* dst;
  const char* src;
  size_t bytes;
};

// The pieces of the segments that go through the staging buffers; the others
// (small ones, and host arrays in pinned memory) are queued on s as they are.
int split_segments(const std::vector<HostSegment>& segs, cudaMemcpyKind kind, cudaStream_t s, std::vector<Piece>* pieces) {
  for (const HostSegment& g : segs) {
    if (g.bytes == 0) continue;
    const bool down = kind == cudaMemcpyDeviceToHost;
    if (g.bytes < kStageMin || is_pinned(down ? g.dst : g.src) ||
        (down && g.bytes < kStageTouched && touched(g.dst, g.bytes))) {
      RR_CUDA(cudaMemcpyAsync(g.dst, g.src, g.bytes, kind, s));
      continue;
    }
    for (size_t off = 0; off < g.bytes; off += kPiece)
      pieces->push_back({static_cast<char*>(g.dst) + off, static_cast<const char*>(g.src) + off,
                         std::min(kPiece, g.bytes - off)});
  }
  return RR_OK;
}

// The context's staging buffers, created at the first staged copy.
int staging_of(rr_ctx* ctx, Staging** out) {
  {
    static std::mutex create_mu;
    std::lock_guard<std::mutex> lk(create_mu);
    if (!ctx->staging) ctx->staging = new Staging();
  }
  Staging& st = *ctx->staging;
  std::lock_guard<std::mutex> lk(st.mu);
  if (st.threads == 0) {
    const int nt = std::max(1, std::min<int>(kMaxStageThreads, (int)std::thread::hardware_concurrency()));
    st.buf.resize(2 * nt, nullptr);
    st.ev.resize(2 * nt, nullptr);
    for (int i = 0; i < 2 * nt; ++i) {
      if (!st.buf[i]) RR_CUDA(cudaHostAlloc(&st.buf[i], kPiece, cudaHostAllocDefault));
      if (!st.ev[i]) RR_CUDA(cudaEventCreateWithFlags(&st.ev[i], cudaEventDisableTiming));
    }
    st.threads = nt;
  }
  *out = &st;
  return RR_OK;
}

// work(w) for every w < nt, on a thread each as far as the system gives them, the
// calling thread doing the rest (an exception must not leave through the C
// entry points); the first error wins.
template <class F>
int run_copies(int nt, const char* what, F work) {
  std::vector<cudaError_t> cerr(nt, cudaSuccess);
  std::vector<std::thread> pool;
  pool.reserve(nt);
  int started = 1;
  try {
    for (; started < nt; ++started) pool.emplace_back([&cerr, &work, w = started] { cerr[w] = work(w); });
  } catch (const std::system_error&) {
  }
  cerr[0] = work(0);
  for (int w = started; w < nt; ++w) cerr[w] = work(w);
  for (std::thread& t : pool) t.join();
  for (int w = 0; w < nt; ++w)
    if (cerr[w] != cudaSuccess) return fail(RR_ECUDA, "staged %s copy failed: %s", what, cudaGetErrorString(cerr[w]));
  return RR_OK;
}

}  // namespace

int upload_host(rr_ctx* ctx, const std::vector<HostSegment>& segs, cudaStream_t s) {
  std::vector<Piece> pieces;
  RR_TRY(split_segments(segs, cudaMemcpyHostToDevice, s, &pieces));
  if (pieces.empty()) return RR_OK;
  Staging* st = nullptr;
  RR_TRY(staging_of(ctx, &st));
  std::lock_guard<std::mutex> lk(st->mu);
  const int nt = std::min<int>(st->threads, (int)pieces.size());
  return run_copies(nt, "host-to-device", [&](int w) {
    cudaError_t e = cudaSetDevice(ctx->device);
    int k = 0;
    for (size_t i = (size_t)w; i < pieces.size() && e == cudaSuccess; i += (size_t)nt, ++k) {
      const int b = 2 * w + (k & 1);
      e = cudaEventSynchronize(st->ev[b]);  // the previous transfer from this buffer is done
      if (e != cudaSuccess) break;
      std::memcpy(st->buf[b], pieces[i].src, pieces[i].bytes);
      e = cudaMemcpyAsync(pieces[i].dst, st->buf[b], pieces[i].bytes, cudaMemcpyHostToDevice, s);
      if (e == cudaSuccess) e = cudaEventRecord(st->ev[b], s);
    }
    return e;
  });
}

int download_host(rr_ctx* ctx, const std::vector<HostSegment>& segs, cudaStream_t s) {
  std::vector<Piece> pieces;
  RR_TRY(split_segments(segs, cudaMemcpyDeviceToHost, s, &pieces));
  if (pieces.empty()) return RR_OK;
  // a context that lives for one call (the workers of a batch) pays for its
  // buffers: about 10 ms, a pageable copy of 32 MB
  if (!ctx->staging && (pieces.size() - 1) * kPiece < kStageNew) {
    for (const Piece& q : pieces) RR_CUDA(cudaMemcpyAsync(q.dst, q.src, q.bytes, cudaMemcpyDeviceToHost, s));
    return RR_OK;
  }
  Staging* st = nullptr;
  RR_TRY(staging_of(ctx, &st));
  std::lock_guard<std::mutex> lk(st->mu);
  const int nt = std::min<int>(st->threads, (int)pieces.size());
  return run_copies(nt, "device-to-host", [&](int w) {
    cudaError_t e = cudaSetDevice(ctx->device);
    // piece k of this thread crosses the bus while piece k - 1 is copied out
    const size_t count = (pieces.size() - (size_t)w + (size_t)nt - 1) / (size_t)nt;
    for (size_t k = 0; k <= count && e == cudaSuccess; ++k) {
      if (k < count) {
        const Piece& q = pieces[(size_t)w + k * (size_t)nt];
        const int b = 2 * w + (int)(k & 1);
        e = cudaEventSynchronize(st->ev[b]);
        if (e == cudaSuccess) e = cudaMemcpyAsync(st->buf[b], q.src, q.bytes, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaEventRecord(st->ev[b], s);
      }
      if (k > 0 && e == cudaSuccess) {
        const Piece& q = pieces[(size_t)w + (k - 1) * (size_t)nt];
        const int b = 2 * w + (int)((k - 1) & 1);
        e = cudaEventSynchronize(st->ev[b]);
        if (e == cudaSuccess) std::memcpy(q.dst, st->buf[b], q.bytes);
      }
    }
    return e;
  });
}

}  // namespace rr
