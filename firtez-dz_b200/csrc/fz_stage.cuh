// Large copies from pageable host arrays to the device, included by
// fz_cuda.cu.
//
// A copy from pageable memory runs at the speed of the one thread in which
// the runtime moves it through its own staging (10 GB/s measured, against 53
// GB/s of the link).  Here several threads move pieces of the caller's arrays
// into a ring of pinned buffers and the calling thread, the only one that
// talks to the runtime (a thread's first call to it costs about 0.1 ms),
// sends each on: 55 MB in 1.4 ms instead of 5.5.  The pieces are written past
// the caches: read back out of a core's cache the link gave 24 GB/s, and the
// same copy took 2.4 ms.  Four threads fill the link (six or eight gain 0.05
// ms), and pieces of 512 KB cost half the calls of 256 KB ones (1.4 against
// 1.9 ms).
//
// The ring (4 MB) belongs to one object and is freed with it; the threads live
// for one call.  Pinning it takes 2 to 5 ms (8 MB up to 9), so an object gets
// it once its copies have added up to STAGE_BUY, which by themselves cost as
// much: a few small copies never pay for a ring.  Below STAGE_MIN, starting
// the threads (0.1 ms) and a first piece (0.1 ms) take most of what they save,
// and where the ring cannot be had the plain copy does the work.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace fzstage {

constexpr int STAGE_THREADS = 4, STAGE_SLOTS = 8;
constexpr size_t STAGE_PIECE = (size_t)512 << 10, STAGE_MIN = (size_t)4 << 20, STAGE_BUY = (size_t)32 << 20;

struct Seg {   // one array
  void* dev;
  const void* host;
  size_t bytes;
};

// n bytes to a 16-byte aligned buffer, past the caches
inline void stream_copy(unsigned char* dst, const unsigned char* src, size_t n) {
  size_t m = 0;
#if defined(__SSE2__)
  for (; m + 64 <= n; m += 64) {
    __m128i v[4];
    for (int k = 0; k < 4; ++k) v[k] = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + m + 16 * k));
    for (int k = 0; k < 4; ++k) _mm_stream_si128(reinterpret_cast<__m128i*>(dst + m + 16 * k), v[k]);
  }
  _mm_sfence();
#endif
  std::memcpy(dst + m, src + m, n - m);
}

class HostStage {
 public:
  HostStage() = default;
  HostStage(const HostStage&) = delete;
  HostStage& operator=(const HostStage&) = delete;
  ~HostStage() { release(); }

  // The nseg arrays to the device, in order on s with what is enqueued there;
  // the host arrays may change once this returns.
  cudaError_t upload(cudaStream_t s, const Seg* segs, int nseg) {
    std::lock_guard<std::mutex> lock(mu_);
    size_t total = 0;
    for (int i = 0; i < nseg; ++i) total += segs[i].bytes;
    std::vector<Piece> pieces;
    if (!buf_) moved_ += total;
    bool staged = total >= STAGE_MIN && (buf_ || moved_ >= STAGE_BUY) && reserve();
    if (staged) {
      try {
        pieces.reserve(total / STAGE_PIECE + nseg);
      } catch (const std::exception&) {
        staged = false;
      }
    }
    if (!staged) {
      for (int i = 0; i < nseg; ++i) {
        const cudaError_t e = cudaMemcpyAsync(segs[i].dev, segs[i].host, segs[i].bytes, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
      }
      return cudaStreamSynchronize(s);   // then the sources have been read
    }
    for (int i = 0; i < nseg; ++i)
      for (size_t o = 0; o < segs[i].bytes; o += STAGE_PIECE)   // within the reserved capacity
        pieces.push_back({(unsigned char*)segs[i].dev + o, (const unsigned char*)segs[i].host + o,
                          std::min(STAGE_PIECE, segs[i].bytes - o)});
    return run(s, pieces);
  }

 private:
  struct Piece {
    unsigned char* dev;
    const unsigned char* host;
    size_t n;
  };
  std::mutex mu_;   // one copy at a time: the ring is the object's
  unsigned char* buf_ = nullptr;
  size_t moved_ = 0;   // bytes copied before the ring was there
  cudaEvent_t ev_[STAGE_SLOTS] = {};   // a slot's last copy

  void release() {
    for (cudaEvent_t& e : ev_)
      if (e) cudaEventSynchronize(e), cudaEventDestroy(e), e = nullptr;
    if (buf_) cudaFreeHost(buf_);
    buf_ = nullptr;
  }

  bool reserve() {
    if (buf_) return true;
    if (cudaMallocHost(&buf_, STAGE_SLOTS * STAGE_PIECE) == cudaSuccess) {
      bool ok = true;
      for (cudaEvent_t& e : ev_) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
      if (ok) return true;
    }
    cudaGetLastError();   // not this copy's failure
    release();
    return false;
  }

  // Piece i goes through slot i % STAGE_SLOTS.  Threads claim pieces in
  // order, wait until the slot's last piece has left (free) and fill it; the
  // caller sends pieces in order as they are ready and, while the next one
  // is not, retires sent ones.  With no thread at all the caller fills too.
  cudaError_t run(cudaStream_t s, const std::vector<Piece>& pieces) {
    const size_t np = pieces.size();
    for (cudaEvent_t e : ev_) {   // the previous upload's pieces
      const cudaError_t r = cudaEventSynchronize(e);
      if (r != cudaSuccess) return r;
    }
    std::atomic<size_t> next{0}, retired{0};   // claimed; pieces before `retired` have left their slots
    std::atomic<size_t> ready[STAGE_SLOTS];    // 1 + the piece a slot holds
    for (auto& r : ready) r.store(0);
    std::atomic<bool> stop{false};
    auto fill = [&](size_t i) {
      stream_copy(buf_ + (i % STAGE_SLOTS) * STAGE_PIECE, pieces[i].host, pieces[i].n);
      ready[i % STAGE_SLOTS].store(i + 1, std::memory_order_release);
    };
    auto work = [&] {
      for (size_t i; (i = next.fetch_add(1)) < np;) {
        while (i >= retired.load(std::memory_order_acquire) + STAGE_SLOTS) {
          if (stop.load()) return;
          std::this_thread::yield();
        }
        fill(i);
      }
    };
    std::thread th[STAGE_THREADS];
    const int hw = (int)std::thread::hardware_concurrency();
    const int want = std::min(STAGE_THREADS, hw - 1);
    int nt = 0;
    try {
      for (; nt < want; ++nt) th[nt] = std::thread(work);
    } catch (const std::exception&) {   // fewer threads, then
    }
    cudaError_t e = cudaSuccess;
    size_t sent = 0, done = 0;
    while (sent < np && e == cudaSuccess) {
      if (done < sent) {
        const cudaError_t q = cudaEventQuery(ev_[done % STAGE_SLOTS]);
        if (q == cudaSuccess)
          retired.store(++done, std::memory_order_release);
        else if (q != cudaErrorNotReady)
          e = q;
      }
      if (nt == 0 && sent < done + STAGE_SLOTS) fill(sent);
      if (e == cudaSuccess && ready[sent % STAGE_SLOTS].load(std::memory_order_acquire) == sent + 1) {
        const Piece& p = pieces[sent];
        e = cudaMemcpyAsync(p.dev, buf_ + (sent % STAGE_SLOTS) * STAGE_PIECE, p.n, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaEventRecord(ev_[sent % STAGE_SLOTS], s);
        ++sent;
      }
    }
    stop.store(true);
    for (int k = 0; k < nt; ++k) th[k].join();
    if (cudaPeekAtLastError() == cudaErrorNotReady) cudaGetLastError();   // of the queries, not an error
    return e;
  }
};

}  // namespace fzstage
