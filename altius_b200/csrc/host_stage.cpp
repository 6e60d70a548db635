#include "host_stage.h"

#include <algorithm>
#include <cstring>
#include <exception>
#include <map>
#include <new>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace ac {
namespace {
// Non-temporal stores: the link then reads the ring from memory, at its full rate. Chunks written with
// plain stores sit in the caches of the core that wrote them, and reading them back from there holds
// the link at 18 GB/s (19 MB with four threads: 1060 us, against 480 this way).
void copy_past_caches(char* dst, const char* src, size_t bytes) {
#if defined(__x86_64__)
  size_t i = 0;
  for (; i + 64 <= bytes; i += 64) {
    const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i)), b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 16)),
                  c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 32)), d = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 48));
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i), a);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 16), b);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 32), c);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 48), d);
  }
  if (i < bytes) std::memcpy(dst + i, src + i, bytes - i);
  _mm_sfence();
#else
  std::memcpy(dst, src, bytes);
#endif
}

inline void relax() {
#if defined(__x86_64__)
  _mm_pause();
#else
  std::this_thread::yield();
#endif
}
}  // namespace

std::shared_ptr<HostStage> HostStage::of_device(int device) {
  static std::mutex m;
  static std::map<int, std::weak_ptr<HostStage>> made;
  // Nothing may be thrown through the C interface: without memory for it the caller does without.
  try {
    std::lock_guard<std::mutex> lock(m);
    if (std::shared_ptr<HostStage> s = made[device].lock()) return s;
    std::shared_ptr<HostStage> s(new HostStage());
    if (!s->init()) return nullptr;
    made[device] = s;
    return s;
  } catch (const std::exception&) {
    return nullptr;
  }
}

bool HostStage::init() {
  if (cudaHostAlloc(reinterpret_cast<void**>(&ring_), kChunk * kSlots, cudaHostAllocPortable) != cudaSuccess) {
    (void)cudaGetLastError();
    ring_ = nullptr;
    return false;
  }
  for (cudaEvent_t& e : left_)
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
  const int cores = (int)std::max(1u, std::thread::hardware_concurrency());
  // Without (all of) them the uploading thread copies what nobody else has taken.
  try {
    for (int i = 0; i < std::min(4, cores / 2); ++i) threads_.emplace_back([this] { worker(); });
  } catch (const std::exception&) {
  }
  return true;
}

HostStage::~HostStage() {
  {
    std::lock_guard<std::mutex> lock(m_);
    stop_ = true;
  }
  cv_.notify_all();
  for (std::thread& t : threads_) t.join();
  for (cudaEvent_t e : left_)
    if (e) cudaEventDestroy(e);
  if (ring_) cudaFreeHost(ring_);
}

// Copies the next piece of a chunk below `limit` whose slot is free; false if there is none now.
bool HostStage::copy_next(int limit) {
  int i = next_.load(std::memory_order_relaxed);
  const int c = i / kPieces;
  if (c >= limit || c >= allowed_.load(std::memory_order_acquire)) return false;
  if (!next_.compare_exchange_strong(i, i + 1)) return false;
  constexpr size_t kPiece = kChunk / kPieces;
  const size_t in = (size_t)(i % kPieces) * kPiece, at = (size_t)c * kChunk + in;
  if (at < bytes_) copy_past_caches(ring_ + (size_t)(c % kSlots) * kChunk + in, src_ + at, std::min(kPiece, bytes_ - at));
  done_[c].fetch_add(1, std::memory_order_release);
  return true;
}

void HostStage::worker() {
  uint64_t seen = 0;
  for (;;) {
    {
      std::unique_lock<std::mutex> lock(m_);
      cv_.wait(lock, [&] { return stop_ || job_ != seen; });
      if (stop_) return;
      seen = job_;
      ++busy_;
    }
    while (next_.load(std::memory_order_relaxed) < chunks_ * kPieces)
      if (!copy_next(chunks_)) relax();
    std::lock_guard<std::mutex> lock(m_);
    --busy_;
  }
}

cudaError_t HostStage::upload(void* dst, const void* src, size_t bytes, cudaStream_t st, const std::function<cudaError_t(size_t)>& sent) {
  auto whole = [&] {
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    return e == cudaSuccess && sent ? sent(bytes) : e;
  };
  // While another thread's upload holds the ring this one takes the driver's path: both then run at once.
  std::unique_lock<std::mutex> use(use_, std::try_to_lock);
  if (!use.owns_lock()) return whole();
  const int n = (int)((bytes + kChunk - 1) / kChunk);
  std::unique_ptr<std::atomic<char>[]> more;
  if (done_size_ < n) {                       // only ever changed under use_
    more.reset(new (std::nothrow) std::atomic<char>[n]);
    if (!more) return whole();
  }
  for (cudaEvent_t e : left_)                 // slots an earlier upload may still occupy
    if (cudaError_t err = cudaEventSynchronize(e)) return err;
  {
    // Workers that have not left the previous job yet (all its chunks are taken: soon).
    std::unique_lock<std::mutex> lock(m_);
    while (busy_ > 0) {
      lock.unlock();
      relax();
      lock.lock();
    }
    if (more) {
      done_ = std::move(more);
      done_size_ = n;
    }
    for (int i = 0; i < n; ++i) done_[i].store(0, std::memory_order_relaxed);
    src_ = static_cast<const char*>(src);
    bytes_ = bytes;
    chunks_ = n;
    next_.store(0);
    allowed_.store(std::min(n, kSlots));
    ++job_;
  }
  cv_.notify_all();
  cudaError_t err = cudaSuccess;
  int allowed = std::min(n, kSlots);
  for (int c = 0; c < n && err == cudaSuccess; ++c) {
    do {
      // Chunk allowed - kSlots is on its way (it is below c): once it has left, its slot is free.
      while (allowed < n && allowed - kSlots < c) {
        const cudaError_t left = cudaEventQuery(left_[allowed % kSlots]);
        if (left != cudaSuccess) {
          (void)cudaGetLastError();
          if (left != cudaErrorNotReady) err = left;   // a fault on the device: the slot never gets free
          break;
        }
        allowed_.store(++allowed, std::memory_order_release);
      }
      if (err != cudaSuccess) break;
      if (!copy_next(c + 1)) relax();         // this chunk itself, if no worker has taken it yet
    } while (done_[c].load(std::memory_order_acquire) < kPieces);
    if (err != cudaSuccess) break;
    const size_t at = (size_t)c * kChunk;
    err = cudaMemcpyAsync(static_cast<char*>(dst) + at, ring_ + (size_t)(c % kSlots) * kChunk, std::min(kChunk, bytes - at),
                          cudaMemcpyHostToDevice, st);
    if (err == cudaSuccess) err = cudaEventRecord(left_[c % kSlots], st);
    if (err == cudaSuccess && sent) err = sent(std::min(bytes, at + kChunk));
  }
  if (err != cudaSuccess) {                   // nobody may go on reading the caller's memory
    next_.store(n * kPieces);
    for (;;) {
      std::lock_guard<std::mutex> lock(m_);
      if (busy_ == 0) break;
    }
  }
  return err;
}

}  // namespace ac
