// Device context: stream, buffer cache, scratch, error word.
#include "device.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace bsz {

DevStream::~DevStream() {
  if (dev && p) dev->release(this);
}

Device::Device(int ordinal) : ordinal_(ordinal) {
  BSZ_CUDA(cudaSetDevice(ordinal));
  cudaDeviceProp prop;
  BSZ_CUDA(cudaGetDeviceProperties(&prop, ordinal));
  if (prop.major < 10)
    throw CudaError("bitstreamzoo_b200 needs an sm_100 (Blackwell B200) device; device " +
                    std::to_string(ordinal) + " is " + prop.name);
  sm_count_ = prop.multiProcessorCount;
  BSZ_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
  void* err = nullptr;
  BSZ_CUDA(cudaHostAlloc(&err, 64, cudaHostAllocMapped));
  std::memset(err, 0, 64);
  err_ = err_now_ = static_cast<uint32_t*>(err);
}

Device::~Device() {
  cudaSetDevice(ordinal_);
  if (stream_) cudaStreamSynchronize(stream_);
  for (auto& kv : all_) cudaFree(kv.first);
  if (d_scan_) cudaFree(d_scan_);
  if (err_) cudaFreeHost(err_);
  for (auto& pool : events_)
    for (cudaEvent_t e : pool) cudaEventDestroy(e);
  if (d_scratch_) cudaFree(d_scratch_);
  arena_.reset();
  for (auto& kv : pinned_->free) cudaFreeHost(kv.second);
  pinned_->free.clear();
  copies_.reset();
  if (stream_) cudaStreamDestroy(stream_);
}

// Cached blocks: a run takes up to a few dozen, of some hundred KiB at most.
constexpr size_t kMaxPinnedFree = 512, kMaxPinnedBytes = size_t(64) << 20;

std::shared_ptr<void> Device::pinned_block(size_t bytes) {
  bytes = std::max<size_t>(4096, (bytes + 4095) / 4096 * 4096);
  void* p = nullptr;
  size_t have = bytes;
  auto it = pinned_->free.lower_bound(bytes);
  if (it != pinned_->free.end() && it->first <= 4 * bytes) {
    have = it->first;
    p = it->second;
    pinned_->free.erase(it);
    pinned_->bytes -= have;
  } else {
    BSZ_CUDA(cudaHostAlloc(&p, bytes, cudaHostAllocDefault));
  }
  // the cache outlives the Device only through blocks still referenced:
  // those are freed directly when the Device is gone
  std::weak_ptr<PinnedCache> cache = pinned_;
  return std::shared_ptr<void>(p, [cache, have](void* q) {
    auto c = cache.lock();
    if (c && c->free.size() < kMaxPinnedFree && c->bytes + have <= kMaxPinnedBytes) {
      c->free.emplace(have, q);
      c->bytes += have;
    } else {
      cudaFreeHost(q);
    }
  });
}

// Copies between pageable host memory and the device.  A chunk passes through
// one of a ring of page-locked buffers: worker threads do the memcpys (and
// take the page faults of a fresh destination) several at a time, the calling
// thread issues the DMAs, in order.  One thread alone copies at about 10 GB/s,
// a fifth of the link; two 32 MiB chunks left a 16 MiB stream with no overlap
// at all (MatchStar of 2^27 bits from and to host memory on a B200: 4.1 ms a
// call).
constexpr size_t kCopyChunk = size_t(1) << 20;
constexpr size_t kCopyRing = 24;
constexpr size_t kDirectBytes = size_t(1) << 20;
constexpr unsigned kCopyWorkers = 8;

// memcpy into a DMA buffer (16-byte aligned) past the caches: the DMA reads
// lines that lie modified in several cores' caches at 12 GB/s, lines in memory
// at 40.
void stream_copy(char* dst, const char* src, size_t n) {
#if defined(__SSE2__)
  size_t i = 0;
  for (; i + 64 <= n; i += 64) {
    const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i));
    const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 16));
    const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 32));
    const __m128i d = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 48));
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i), a);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 16), b);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 32), c);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 48), d);
  }
  _mm_sfence();
  if (i < n) std::memcpy(dst + i, src + i, n - i);
#else
  std::memcpy(dst, src, n);
#endif
}

class CopyPool {
 public:
  CopyPool(int ordinal, cudaStream_t stream) : ordinal_(ordinal), stream_(stream) {
    const unsigned n = std::max(1u, std::min(kCopyWorkers, std::thread::hardware_concurrency()));
    threads_.reserve(n);
    try {
      BSZ_CUDA(cudaHostAlloc(&block_, kCopyRing * kCopyChunk, cudaHostAllocDefault));
      for (cudaEvent_t& e : ev_) BSZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      // where the process may start no more threads, those it got do
      for (unsigned i = 0; i < n; ++i) try {
          threads_.emplace_back([this] { serve(); });
        } catch (const std::system_error&) {
          if (threads_.empty()) throw;
          break;
        }
    } catch (...) {
      release();
      throw;
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : threads_) t.join();
    release();
  }
  CopyPool(const CopyPool&) = delete;
  CopyPool& operator=(const CopyPool&) = delete;

  // Returns when every chunk has been handed to the stream (to the device:
  // `src` may be reused) or has arrived (to the host).
  void copy(void* dst, const void* src, size_t bytes, bool to_host) {
    const size_t chunks = (bytes + kCopyChunk - 1) / kCopyChunk;
    // buffers may still be in flight to the device from an earlier copy
    for (cudaEvent_t e : ev_) BSZ_CUDA(cudaEventSynchronize(e));
    {
      std::lock_guard<std::mutex> lk(mu_);
      dst_ = static_cast<char*>(dst);
      src_ = static_cast<const char*>(src);
      bytes_ = bytes;
      chunks_ = chunks;
      to_host_ = to_host;
      next_ = 0;
      issued_ = 0;
      failed_ = false;
      for (auto& c : copied_) c = 0;
      busy_ = threads_.size();
      ++job_;
    }
    wake_.notify_all();
    std::exception_ptr error;
    try {
      for (size_t c = 0; c < chunks && !failed_; ++c) {
        const size_t off = c * kCopyChunk, len = std::min(kCopyChunk, bytes - off), b = c % kCopyRing;
        // the workers' part of this buffer: filled with chunk c, or chunk
        // c - kCopyRing copied out (each counts the buffer's copies)
        const size_t want = c / kCopyRing + (to_host ? 0 : 1);
        while (copied_[b].load(std::memory_order_acquire) < want && !failed_) std::this_thread::yield();
        if (to_host)
          BSZ_CUDA(cudaMemcpyAsync(buffer(b), src_ + off, len, cudaMemcpyDeviceToHost, stream_));
        else
          BSZ_CUDA(cudaMemcpyAsync(dst_ + off, buffer(b), len, cudaMemcpyHostToDevice, stream_));
        BSZ_CUDA(cudaEventRecord(ev_[b], stream_));
        issued_.store(c + 1, std::memory_order_release);
      }
    } catch (...) {
      error = std::current_exception();
      failed_ = true;
    }
    std::unique_lock<std::mutex> lk(mu_);
    done_.wait(lk, [this] { return busy_ == 0; });
    if (error) std::rethrow_exception(error);
    if (failed_) throw CudaError("copy between host and device failed");
  }

 private:
  int ordinal_;
  cudaStream_t stream_;
  void* block_ = nullptr;
  cudaEvent_t ev_[kCopyRing] = {};             // a buffer's last DMA
  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable wake_, done_;
  uint64_t job_ = 0;
  size_t busy_ = 0;
  bool stop_ = false, to_host_ = false;
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t bytes_ = 0, chunks_ = 0;
  std::atomic<size_t> next_{0}, issued_{0};
  std::atomic<size_t> copied_[kCopyRing] = {};   // memcpys done with each buffer in this job
  std::atomic<bool> failed_{false};

  void release() {
    for (cudaEvent_t e : ev_)
      if (e) cudaEventDestroy(e);
    if (block_) cudaFreeHost(block_);
  }

  char* buffer(size_t b) const { return static_cast<char*>(block_) + b * kCopyChunk; }

  void serve() {
    cudaSetDevice(ordinal_);
    uint64_t seen = 0;
    while (true) {
      {
        std::unique_lock<std::mutex> lk(mu_);
        wake_.wait(lk, [&] { return stop_ || job_ != seen; });
        if (stop_) return;
        seen = job_;
      }
      work();
      bool last;
      {
        std::lock_guard<std::mutex> lk(mu_);
        last = --busy_ == 0;
      }
      if (last) done_.notify_one();
    }
  }

  void work() {
    for (size_t c; (c = next_.fetch_add(1)) < chunks_ && !failed_;) {
      const size_t off = c * kCopyChunk, len = std::min(kCopyChunk, bytes_ - off), b = c % kCopyRing;
      // the DMA that this memcpy waits for: into the buffer (to the host), or
      // the one that read it a ring ago
      const size_t dma = to_host_ ? c + 1 : c < kCopyRing ? 0 : c - kCopyRing + 1;
      while (issued_.load(std::memory_order_acquire) < dma && !failed_) std::this_thread::yield();
      if (failed_) return;
      if (dma > 0 && cudaEventSynchronize(ev_[b]) != cudaSuccess) {
        failed_ = true;
        return;
      }
      if (to_host_) std::memcpy(dst_ + off, buffer(b), len);
      else stream_copy(buffer(b), src_ + off, len);
      copied_[b].fetch_add(1, std::memory_order_release);
    }
  }
};

CopyPool& Device::copy_pool() {
  if (!copies_) copies_ = std::make_unique<CopyPool>(ordinal_, stream_);
  return *copies_;
}

void Device::h2d(void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return;
  if (bytes <= kDirectBytes)
    BSZ_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream_));
  else
    copy_pool().copy(dst, src, bytes, false);
}

void Device::d2h(void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return;
  if (bytes <= kDirectBytes) {
    BSZ_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream_));
    BSZ_CUDA(cudaStreamSynchronize(stream_));
  } else {
    copy_pool().copy(dst, src, bytes, true);
  }
}

void* Device::raw_alloc(size_t bytes) {
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    trim_cache();
    e = cudaMalloc(&p, bytes);
  }
  if (e != cudaSuccess)
    throw CudaError(std::string("cudaMalloc(") + std::to_string(bytes) +
                    ") failed: " + cudaGetErrorString(e) +
                    (e == cudaErrorMemoryAllocation ? " (out of memory)" : ""));
  ++n_mallocs;
  all_.push_back({p, bytes});
  return p;
}

BufRef Device::alloc_stream(int64_t n_words) {
  // Round to 256 bytes so vector loops may run over whole 16-byte pairs.
  size_t bytes = (static_cast<size_t>(std::max<int64_t>(n_words, 1)) * 8 + 255) & ~size_t(255);
  void* p = nullptr;
  auto it = free_.find(bytes);
  if (it != free_.end()) {
    p = it->second;
    free_.erase(it);
  } else {
    p = raw_alloc(bytes);
  }
  auto s = std::make_shared<DevStream>();
  s->p = static_cast<uint64_t*>(p);
  s->n_words = n_words;
  s->bytes = bytes;
  s->dev = this;
  bytes_live += static_cast<int64_t>(bytes);
  bytes_peak = std::max(bytes_peak, bytes_live);
  return s;
}

constexpr size_t kArenaBytes = size_t(256) << 10;

std::shared_ptr<void> Device::host_slice(size_t bytes) {
  bytes = (bytes + 255) & ~size_t(255);
  if (bytes > kArenaBytes / 4) return pinned_block(bytes);
  if (!arena_ || arena_used_ + bytes > kArenaBytes) {
    arena_ = pinned_block(kArenaBytes);
    arena_used_ = 0;
  }
  char* p = static_cast<char*>(arena_.get()) + arena_used_;
  arena_used_ += bytes;
  return std::shared_ptr<void>(arena_, p);
}

BufRef Device::host_stream(const uint64_t* words, int64_t have, int64_t n_words, uint64_t fill) {
  auto s = std::make_shared<DevStream>();
  s->host = host_slice(static_cast<size_t>(std::max<int64_t>(n_words, 1)) * 8);
  s->p = static_cast<uint64_t*>(s->host.get());
  s->n_words = n_words;
  if (have > 0) std::memcpy(s->p, words, static_cast<size_t>(have) * 8);
  for (int64_t w = have; w < n_words; ++w) s->p[w] = fill;
  return s;
}

void Device::read_stream(const BufRef& b, int64_t n, uint64_t* out) {
  const void* at_host = b->host ? b->p : b->mirror.get();
  if (at_host) std::memcpy(out, at_host, static_cast<size_t>(n) * 8);
  else d2h(out, b->p, static_cast<size_t>(n) * 8);
}

void Device::release(DevStream* s) {
  free_.emplace(s->bytes, s->p);
  bytes_live -= static_cast<int64_t>(s->bytes);
  s->p = nullptr;
}

void Device::trim_cache() {
  cudaStreamSynchronize(stream_);
  for (auto& kv : free_) {
    cudaFree(kv.second);
    all_.erase(std::remove_if(all_.begin(), all_.end(),
                              [&](const std::pair<void*, size_t>& a) { return a.first == kv.second; }),
               all_.end());
  }
  free_.clear();
}

uint32_t* Device::scan_state(int64_t n_u32) {
  if (n_u32 > scan_cap_) {
    if (d_scan_) {
      BSZ_CUDA(cudaStreamSynchronize(stream_));
      BSZ_CUDA(cudaFree(d_scan_));
    }
    int64_t cap = std::max<int64_t>(n_u32, 4096);
    BSZ_CUDA(cudaMalloc(&d_scan_, static_cast<size_t>(cap) * 4));
    ++n_mallocs;
    scan_cap_ = cap;
  }
  BSZ_CUDA(cudaMemsetAsync(d_scan_, 0, static_cast<size_t>(n_u32) * 4, stream_));
  return d_scan_;
}

void* Device::scratch(size_t bytes) {
  if (bytes > scratch_cap_) {
    if (d_scratch_) {
      BSZ_CUDA(cudaStreamSynchronize(stream_));
      BSZ_CUDA(cudaFree(d_scratch_));
    }
    size_t cap = std::max<size_t>(bytes, 1 << 16);
    BSZ_CUDA(cudaMalloc(&d_scratch_, cap));
    ++n_mallocs;
    scratch_cap_ = cap;
  }
  return d_scratch_;
}

uint32_t Device::take_error() {
  BSZ_CUDA(cudaStreamSynchronize(stream_));
  const uint32_t h = *reinterpret_cast<volatile uint32_t*>(err_);
  if (h) *reinterpret_cast<volatile uint32_t*>(err_) = 0;
  return h;
}

cudaEvent_t Device::take_event(bool timing) {
  auto& pool = events_[timing];
  if (!pool.empty()) {
    cudaEvent_t e = pool.back();
    pool.pop_back();
    return e;
  }
  cudaEvent_t e;
  BSZ_CUDA(cudaEventCreateWithFlags(&e, timing ? cudaEventDefault : cudaEventDisableTiming));
  return e;
}

void Device::give_event(cudaEvent_t e, bool timing) {
  auto& pool = events_[timing];
  if (pool.size() < 64) pool.push_back(e);
  else cudaEventDestroy(e);
}

void Device::sync() {
  BSZ_CUDA(cudaStreamSynchronize(stream_));
  BSZ_CUDA(cudaGetLastError());
}

cudaEvent_t Device::prof_event() {
  if (!prof_pool_.empty()) {
    cudaEvent_t e = prof_pool_.back();
    prof_pool_.pop_back();
    return e;
  }
  cudaEvent_t e;
  BSZ_CUDA(cudaEventCreate(&e));
  return e;
}

cudaEvent_t Device::prof_begin() {
  cudaEvent_t e = prof_event();
  BSZ_CUDA(cudaEventRecord(e, stream_));
  return e;
}

void Device::prof_end(const char* name, cudaEvent_t begin) {
  cudaEvent_t e = prof_event();
  BSZ_CUDA(cudaEventRecord(e, stream_));
  prof_pending_.push_back({name, begin, e});
  if (prof_pending_.size() > 4096) prof_report();   // resolve in batches
}

std::string Device::prof_report() {
  BSZ_CUDA(cudaStreamSynchronize(stream_));
  for (auto& r : prof_pending_) {
    float ms = 0;
    cudaEventElapsedTime(&ms, r.a, r.b);
    auto& t = prof_totals_[r.name];
    t.first += 1;
    t.second += ms;
    prof_pool_.push_back(r.a);
    prof_pool_.push_back(r.b);
  }
  prof_pending_.clear();
  std::string js = "{";
  bool first = true;
  for (auto& kv : prof_totals_) {
    char buf[256];
    std::snprintf(buf, sizeof buf, "%s\"%s\":{\"launches\":%lld,\"ms\":%.6f}", first ? "" : ",",
                  kv.first.c_str(), static_cast<long long>(kv.second.first), kv.second.second);
    js += buf;
    first = false;
  }
  return js + "}";
}

void Device::prof_reset() {
  prof_report();
  prof_totals_.clear();
}

}  // namespace bsz
