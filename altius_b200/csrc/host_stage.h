// Uploads of large pageable host buffers. cudaMemcpyAsync from pageable memory copies through the
// driver's own page-locked buffer on the calling thread: 16-19 GB/s on the host measured, a third of
// the link (19 MB: 1080 us, against 359 us from page-locked memory). Here a few threads copy chunks
// into a page-locked ring (past the caches, see the copy) while the chunks in front are on the
// link, so the upload runs at the link's rate after the first chunk.
//
// One stage per device, shared by the sessions that need it and freed with the last of them; one
// upload at a time, and those that find it taken are copied by the driver.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <functional>
#include <condition_variable>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace ac {

class HostStage {
 public:
  // The stage of the current device (its ordinal given), made on first use; null if its memory
  // cannot be had (the caller then lets the driver copy).
  static std::shared_ptr<HostStage> of_device(int device);
  ~HostStage();
  // Enqueues dst (device) <- src (pageable host) on `st`; src has been read when this returns. `sent(n)` is called when
  // the first n bytes have been enqueued, n growing to `bytes`; an error it returns ends the upload.
  cudaError_t upload(void* dst, const void* src, size_t bytes, cudaStream_t st, const std::function<cudaError_t(size_t)>& sent = nullptr);

 private:
  static constexpr size_t kChunk = size_t(1) << 20;
  static constexpr int kPieces = 4;           // a chunk is copied by several threads, so that the first is on its way after 25 us
                                              // (whole chunks: 38 MB 980 us behind the device time, this way 860)
  static constexpr int kSlots = 12;
  HostStage() = default;
  bool init();
  void worker();
  bool copy_next(int limit);

  char* ring_ = nullptr;
  cudaEvent_t left_[kSlots] = {};             // the chunk in this slot is on the device
  std::vector<std::thread> threads_;
  std::mutex use_;                            // one upload at a time
  std::mutex m_;
  std::condition_variable cv_;
  uint64_t job_ = 0;                          // guarded by m_
  int busy_ = 0;                              // workers inside the current job, guarded by m_
  bool stop_ = false;
  const char* src_ = nullptr;
  size_t bytes_ = 0;
  int chunks_ = 0;
  std::atomic<int> next_{0}, allowed_{0};     // next piece to copy; chunks below `allowed_` have a free slot
  std::unique_ptr<std::atomic<char>[]> done_;   // pieces of a chunk that have been copied
  int done_size_ = 0;
};

}  // namespace ac
