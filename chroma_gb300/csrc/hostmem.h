// Host side of the calls that return their results in host buffers.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <functional>
#include <thread>
#include <utility>
#include <vector>

namespace gbc {

// Makes the pages of result buffers resident on other threads while the device works.  A caller's
// fresh buffer (calloc, np.zeros) has no pages, and on GB300's host, whose pages the GPU reads and writes
// through the CPU's page tables, whoever comes first pays for them.  302 MB, measured: a copy from the device
// into resident pages 1.7 ms, into fresh ones 11.5 ms; into pages that a copy to the device has read
// before they were written, and which therefore map the kernel's zero page, 70 to 110 ms (every page is
// replaced under the GPU's translation caches).  Populating for writing takes 10 ms for 302 MB of fresh
// pages on one thread and 4 ms on four (eight were slower), 1.2 ms if they are all there.  It leaves the
// contents alone, so a call that fails leaves the caller's buffer as it was.  (Storing a byte to each page
// from 8 threads takes 2.4 ms, but spoils the buffer before the call has a result for it.)
// Nothing outlives the object; where a page cannot be had this way the copy meets it as before.
class PageTouch {
 public:
  using Ranges = std::vector<std::pair<void*, size_t>>;
  ~PageTouch() { join(); }
  // Makes the pages present and writable, contents unchanged, on `threads` (at most kThreads) helpers;
  // `then` (optional, must not throw) runs on the last of them afterwards, or in join() if one could not
  // be started.
  void populate(Ranges ranges, std::function<void()> then = nullptr, int threads = 1);
  void join();
  static constexpr int kThreads = 4;

 private:
  std::thread th_[kThreads];
  std::atomic<int> left_{0};  // helpers that have not finished
  std::function<void()> then_;
};

// whether every page of a buffer is there (25 us for 302 MB); a page that was only read counts too
bool pages_present(const void* p, size_t bytes);

// The results of a call on their way to the caller's buffers, whose pages are made resident meanwhile.
//   kKeep  the device slots hold whatever the call puts there (the whole result, or a buffer that the
//          caller fetched itself)
//   kLoad  the buffers' contents go to the slots first, on the copy stream: the sites that the call
//          does not own come back unchanged
// Each slot is copied back on the copy stream once the work stream has filled it, beside whatever the
// work stream does next.  Nothing is written to a buffer before its send().
class HostResult {
 public:
  struct Item {
    double* host;
    double* dev;
    size_t bytes;
  };
  enum Mode { kKeep, kLoad };
  // threads: helpers for the pages, more than one where the call is short
  HostResult(cudaStream_t work, cudaStream_t copy, std::vector<Item> items, Mode mode, int threads = 1);
  ~HostResult();
  // from here on the work stream may write the slots
  void ready();
  // slot q -> the caller, after the work enqueued so far
  void send(size_t q);
  // every copy has arrived
  void wait();

 private:
  cudaStream_t work_, copy_;
  std::vector<Item> items_;
  cudaEvent_t ev_ = nullptr;
  int dev_ = 0;
  bool load_ = false, is_ready_ = false;
  cudaError_t err_ = cudaSuccess;
  PageTouch touch_;
};

}  // namespace gbc
