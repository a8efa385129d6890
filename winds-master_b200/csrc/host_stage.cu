// host_stage.cu -- see host_stage.h.
#include "host_stage.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include <sys/mman.h>
#include <unistd.h>

namespace winds {

struct StageLease::Stage {
  int dev = 0;
  cudaStream_t stream = nullptr;
  HostBuf pinned;
  DevBuf scratch;
  std::vector<cudaEvent_t> ev;  // per chunk of a download
  cudaEvent_t used = nullptr;   // after the last DMA from the pinned memory
  bool pending = false;

  // The pinned memory, once no DMA reads it any more. Where the system has none to give
  // (cudaErrorMemoryAllocation, not left behind as the last error) copies go without.
  cudaError_t reserve(size_t bytes) {
    if (pending) {
      const cudaError_t e = cudaEventSynchronize(used);
      if (e != cudaSuccess) return e;
      pending = false;
    }
    if (!pinned.ensure(bytes)) return cudaSuccess;
    cudaGetLastError();
    return cudaErrorMemoryAllocation;
  }
  void destroy() {
    cudaSetDevice(dev);
    if (pending) cudaEventSynchronize(used);
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
    if (used) cudaEventDestroy(used);
    if (stream) cudaStreamDestroy(stream);
    pinned.release();
    scratch.release();
  }
};

namespace {

std::mutex g_mu;
std::vector<StageLease::Stage *> g_free;

constexpr size_t kChunk = 1u << 20;
constexpr size_t kSmallUpload = 1u << 20;
constexpr size_t kDirect = 16u << 20;
constexpr std::chrono::microseconds kSpin{200};

// A part of a span within one chunk of the staging memory.
struct Piece {
  unsigned char *host, *dev;
  size_t off, bytes;
};

// Threads that copy `bytes` out (host_stage.h), at most half the machine's. wide: one
// per MB, up to 8.
int copy_threads(size_t bytes, bool wide) {
  const int hw = (int)std::thread::hardware_concurrency() / 2;
  const int want = wide ? (int)(bytes / kChunk) : bytes <= 8 * kChunk ? 1 : bytes <= kDirect ? 2 : 8;
  return std::max(1, std::min({8, hw, want}));
}

// Whether the page in the middle of these bytes is there, and not made on its first write.
bool resident(const void *p, size_t bytes) {
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), at = (uintptr_t)p + bytes / 2;
  unsigned char r = 0;
  return mincore((void *)(at / page * page), 1, &r) == 0 && (r & 1);
}

bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace

StageLease::StageLease() {
  int dev = 0;
  if ((err_ = cudaGetDevice(&dev)) != cudaSuccess) return;
  {
    std::lock_guard<std::mutex> g(g_mu);
    for (size_t k = 0; k < g_free.size(); ++k)
      if (g_free[k]->dev == dev) {
        st_ = g_free[k];
        g_free.erase(g_free.begin() + k);
        return;
      }
  }
  st_ = new (std::nothrow) Stage();
  if (!st_) {
    err_ = cudaErrorMemoryAllocation;
    return;
  }
  st_->dev = dev;
  err_ = cudaStreamCreateWithFlags(&st_->stream, cudaStreamNonBlocking);
  if (err_ == cudaSuccess) err_ = cudaEventCreateWithFlags(&st_->used, cudaEventDisableTiming);
}

StageLease::~StageLease() {
  if (!st_) return;
  if (err_ == cudaSuccess && st_->pinned.cap <= kMaxPinned + kMaxPinned / 4 + 256 &&
      st_->scratch.cap <= kMaxDev) {
    std::lock_guard<std::mutex> g(g_mu);
    int kept = 0;
    for (const Stage *s : g_free) kept += s->dev == st_->dev;
    try {
      if (kept < kKept) {
        g_free.push_back(st_);
        return;
      }
    } catch (...) {  // no memory for the list: freed like a stage too many
    }
  }
  st_->destroy();
  delete st_;
}

cudaStream_t StageLease::stream() const { return st_->stream; }
DevBuf &StageLease::scratch() { return st_->scratch; }

cudaError_t StageLease::upload(const HostSpan *v, int n, cudaStream_t s) {
  if (err_ != cudaSuccess) return err_;
  size_t total = 0;
  for (int i = 0; i < n; ++i) total += v[i].bytes;
  cudaError_t e = cudaSuccess;
  unsigned char *pin = nullptr;
  if (total <= kSmallUpload) {
    e = st_->reserve(total);
    if (e == cudaSuccess) pin = static_cast<unsigned char *>(st_->pinned.p);
    else if (e != cudaErrorMemoryAllocation) return err_ = e;
    e = cudaSuccess;
  }
  size_t off = 0, from = 0;  // staged; of it, sent
  unsigned char *to = nullptr;
  const auto send = [&] {
    if (off > from && e == cudaSuccess)
      e = cudaMemcpyAsync(to, pin + from, off - from, cudaMemcpyHostToDevice, s);
    from = off;
  };
  for (int i = 0; i < n && e == cudaSuccess; ++i) {
    if (v[i].bytes == 0) continue;
    unsigned char *dev = static_cast<unsigned char *>(v[i].dev);
    if (!pin || !pageable(v[i].host)) {
      e = cudaMemcpyAsync(dev, v[i].host, v[i].bytes, cudaMemcpyHostToDevice, s);
      continue;
    }
    if (off == from || dev != to + (off - from)) {
      send();
      to = dev;
    }
    std::memcpy(pin + off, v[i].host, v[i].bytes);
    off += v[i].bytes;
  }
  send();
  if (off > 0 && e == cudaSuccess) {
    e = cudaEventRecord(st_->used, s);
    st_->pending = true;
  }
  if (e != cudaSuccess) err_ = e;
  return e;
}

cudaError_t StageLease::download(const HostSpan *v, int n, cudaStream_t s, bool wide) {
  if (err_ != cudaSuccess) return err_;
  size_t bytes = 0, there = 0;  // there: to pageable memory with its pages in place
  for (int i = 0; i < n; ++i) bytes += v[i].bytes;
  for (int i = 0; i < n && !wide && bytes > kDirect; ++i)
    if (v[i].bytes && pageable(v[i].host) && resident(v[i].host, v[i].bytes)) there += v[i].bytes;
  const bool direct = there > bytes / 2;
  std::vector<Piece> pieces;
  // up to kMaxPinned bytes of pieces: a DMA per chunk and run of device memory, then
  // the threads copy each chunk once its event has passed. They start before it has,
  // beside the work that the first DMA waits for: kSpin long they look for themselves,
  // as long as the kinematics of a run take (waking eight threads takes 0.3 ms of its
  // 0.9), then they sleep, so that a long sum does not keep eight cores busy.
  const auto round = [&](size_t total) -> cudaError_t {
    if (total == 0) return cudaSuccess;
    cudaError_t r = st_->reserve(total);
    if (r == cudaErrorMemoryAllocation) {
      r = cudaSuccess;
      for (size_t i = 0; i < pieces.size() && r == cudaSuccess; ++i)
        r = cudaMemcpyAsync(pieces[i].host, pieces[i].dev, pieces[i].bytes, cudaMemcpyDeviceToHost, s);
      return r;
    }
    if (r != cudaSuccess) return r;
    unsigned char *pin = static_cast<unsigned char *>(st_->pinned.p);
    const int chunks = (int)((total + kChunk - 1) / kChunk);
    std::vector<int> first(chunks + 1, (int)pieces.size());  // first piece of a chunk
    for (int i = (int)pieces.size() - 1; i >= 0; --i) first[pieces[i].off / kChunk] = i;
    for (int c = 0; c < chunks && r == cudaSuccess; ++c) {
      for (int i = first[c], j; i < first[c + 1] && r == cudaSuccess; i = j) {
        size_t bytes = pieces[i].bytes;
        for (j = i + 1; j < first[c + 1] && pieces[j].dev == pieces[i].dev + bytes; ++j)
          bytes += pieces[j].bytes;
        r = cudaMemcpyAsync(pin + pieces[i].off, pieces[i].dev, bytes, cudaMemcpyDeviceToHost, s);
      }
      if (r == cudaSuccess && c >= (int)st_->ev.size()) {
        cudaEvent_t ev;
        if ((r = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) == cudaSuccess)
          st_->ev.push_back(ev);
      }
      if (r == cudaSuccess) r = cudaEventRecord(st_->ev[c], s);
    }
    if (r != cudaSuccess) return r;
    std::atomic<int> next{0}, ready{0};  // ready: chunks that landed; < 0: a wait failed
    std::mutex mu;
    std::condition_variable landed;
    const auto work = [&] {
      const auto settled = [&](int c) {
        const int k = ready.load(std::memory_order_acquire);
        return k < 0 || k > c;
      };
      for (int c = next.fetch_add(1); c < chunks; c = next.fetch_add(1)) {
        const auto until = std::chrono::steady_clock::now() + kSpin;
        while (!settled(c) && std::chrono::steady_clock::now() < until) std::this_thread::yield();
        if (!settled(c)) {
          std::unique_lock<std::mutex> g(mu);
          landed.wait(g, [&] { return settled(c); });
        }
        if (ready.load(std::memory_order_acquire) < 0) return;
        for (int i = first[c]; i < first[c + 1]; ++i)
          std::memcpy(pieces[i].host, pin + pieces[i].off, pieces[i].bytes);
      }
    };
    std::vector<std::thread> pool;
    const int nthreads = copy_threads(bytes, wide);
    try {
      pool.reserve(nthreads);
      for (int t = 1; t < nthreads; ++t) pool.emplace_back(work);
    } catch (...) {  // fewer threads, or this one alone
    }
    for (int c = 0; c < chunks && r == cudaSuccess; ++c) {
      r = cudaEventSynchronize(st_->ev[c]);
      {
        std::lock_guard<std::mutex> g(mu);
        ready.store(r == cudaSuccess ? c + 1 : -1, std::memory_order_release);
      }
      landed.notify_all();
    }
    if (r == cudaSuccess) work();
    for (std::thread &x : pool) x.join();
    return r;
  };
  cudaError_t e = cudaSuccess;
  try {
    size_t off = 0;
    for (int i = 0; i < n && e == cudaSuccess; ++i) {
      unsigned char *host = static_cast<unsigned char *>(v[i].host);
      unsigned char *dev = static_cast<unsigned char *>(v[i].dev);
      size_t left = v[i].bytes;
      if (left == 0) continue;
      if (direct || !pageable(host)) {
        e = cudaMemcpyAsync(host, dev, left, cudaMemcpyDeviceToHost, s);
        continue;
      }
      while (left > 0 && e == cudaSuccess) {
        if (off == kMaxPinned) {
          e = round(off);
          pieces.clear();
          off = 0;
        }
        const size_t b = std::min({left, kChunk - off % kChunk, kMaxPinned - off});
        pieces.push_back(Piece{host, dev, off, b});
        host += b, dev += b, off += b, left -= b;
      }
    }
    if (e == cudaSuccess) e = round(off);
  } catch (...) {
    e = cudaErrorMemoryAllocation;
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) err_ = e;  // not kept: copies may still be under way
  return e;
}

void release_stages() {
  std::lock_guard<std::mutex> g(g_mu);
  for (StageLease::Stage *s : g_free) {
    s->destroy();
    delete s;
  }
  g_free.clear();
}

}  // namespace winds
