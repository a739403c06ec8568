// Host side of the calls that return their results in host buffers.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <functional>
#include <thread>
#include <utility>
#include <vector>

namespace gbc {

// whether two host buffers of n bytes share any
inline bool overlap(const void* a, const void* b, size_t n) {
  const char *p = static_cast<const char*>(a), *q = static_cast<const char*>(b);
  return p < q + n && q < p + n;
}

// Makes the pages of result buffers resident on another thread while the device works.  A caller's
// fresh buffer (calloc, np.zeros) has no pages, and on GB300's host, whose pages the GPU reads and writes
// through the CPU's page tables, whoever comes first pays for them.  302 MB, measured: a copy from the device
// into resident pages 1.7 ms, into fresh ones 11.5 ms; into pages that a copy to the device has read
// before they were written, and which therefore map the kernel's zero page, 70 to 110 ms (every page is
// replaced under the GPU's translation caches).  Populating for writing takes 10 ms for 302 MB on one
// thread (more threads gain nothing), beside the device's work; stores of one byte per page from 8
// threads take 2 to 3 ms, but only a buffer that the call overwrites entirely may be stored to.
// Nothing outlives the object; where a page cannot be had this way the copy meets it as before.
class PageTouch {
 public:
  using Ranges = std::vector<std::pair<void*, size_t>>;
  ~PageTouch() { join(); }
  // Makes the pages present and writable, contents unchanged; `then` (optional, must not throw) runs on
  // the helper thread afterwards, or in join() if no thread could be started.
  void populate(Ranges ranges, std::function<void()> then = nullptr);
  // For buffers about to be overwritten: one byte of each page is set to zero.
  void overwrite(Ranges ranges);
  void join();

 private:
  std::thread th_[8];
  std::function<void()> then_;
};

// The results of a call on their way to the caller's buffers.  With `load` the buffers' contents go to
// the device slots first, on the copy stream (an odd-sites solve must hand the even sites back
// unchanged); each slot is copied back on the copy stream once the work stream has filled it, beside
// whatever the work stream does next.  `whole`: the call overwrites the buffers entirely.
class HostResult {
 public:
  struct Item {
    double* host;
    double* dev;
    size_t bytes;
  };
  enum Mode { kKeep, kLoad, kWhole };
  HostResult(cudaStream_t work, cudaStream_t copy, std::vector<Item> items, Mode mode);
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
