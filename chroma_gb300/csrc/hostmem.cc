#include "hostmem.h"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <exception>

#include "ctx.h"

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14
#endif

namespace gbc {
namespace {

// below this a buffer's page faults cost less than a thread
constexpr size_t kSmall = 2u << 20;

size_t page_size() {
  const long ps = sysconf(_SC_PAGESIZE);
  return ps > 0 ? (size_t)ps : 4096;
}

size_t total_bytes(const PageTouch::Ranges& ranges) {
  size_t n = 0;
  for (const auto& r : ranges) n += r.second;
  return n;
}

}  // namespace

bool pages_present(const void* p, size_t bytes) {
  const size_t page = page_size();
  const uintptr_t lo = reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)(page - 1);
  const size_t len = reinterpret_cast<uintptr_t>(p) + bytes - lo;
  std::vector<unsigned char> in((len + page - 1) / page);
  if (mincore(reinterpret_cast<void*>(lo), len, in.data()) != 0) return false;
  return std::all_of(in.begin(), in.end(), [](unsigned char b) { return b & 1; });
}

void PageTouch::populate(Ranges ranges, std::function<void()> then, int threads) {
  join();
  then_ = std::move(then);
  const size_t total = total_bytes(ranges);
  if (total < kSmall) return;
  // one per 8 MB: a helper takes some 50 us to start
  const int n = std::min({std::max(threads, 1), (int)kThreads, (int)std::min<size_t>(total / (8u << 20) + 1, kThreads)});
  left_ = n;
  try {
    for (int k = 0; k < n; ++k)
      th_[k] = std::thread([this, ranges, page = page_size(), k, n] {
        for (const auto& r : ranges) {
          const uintptr_t base = reinterpret_cast<uintptr_t>(r.first);
          const uintptr_t p = (base + r.second / n * k) & ~(uintptr_t)(page - 1);
          const uintptr_t end = base + (k + 1 == n ? r.second : r.second / n * (k + 1));
          if (end > p) (void)madvise(reinterpret_cast<void*>(p), end - p, MADV_POPULATE_WRITE);
        }
        if (left_.fetch_sub(1) == 1 && then_) {
          then_();
          then_ = nullptr;
        }
      });
  } catch (const std::exception&) {  // no thread: join() runs `then`
  }
}

void PageTouch::join() {
  for (auto& t : th_)
    if (t.joinable()) t.join();
  if (then_) then_();
  then_ = nullptr;
}

HostResult::HostResult(cudaStream_t work, cudaStream_t copy, std::vector<Item> items, Mode mode, int threads)
    : work_(work), copy_(copy), items_(std::move(items)), load_(mode == kLoad) {
  GBC_CUDA(cudaGetDevice(&dev_));
  GBC_CUDA(cudaEventCreateWithFlags(&ev_, cudaEventDisableTiming));
  PageTouch::Ranges ranges;
  for (const Item& i : items_) ranges.push_back({i.host, i.bytes});
  if (mode == kKeep) {
    touch_.populate(std::move(ranges), nullptr, threads);
  } else {
    // the slots may still be in use by work enqueued before this call
    GBC_CUDA(cudaEventRecord(ev_, work_));
    GBC_CUDA(cudaStreamWaitEvent(copy_, ev_, 0));
    touch_.populate(std::move(ranges), [this] {
      err_ = cudaSetDevice(dev_);
      for (const Item& i : items_)
        if (err_ == cudaSuccess) err_ = cudaMemcpyAsync(i.dev, i.host, i.bytes, cudaMemcpyHostToDevice, copy_);
    }, threads);
  }
}

HostResult::~HostResult() {
  touch_.join();
  cudaStreamSynchronize(copy_);
  if (ev_) cudaEventDestroy(ev_);
}

void HostResult::ready() {
  if (is_ready_) return;
  is_ready_ = true;
  touch_.join();
  GBC_CUDA(err_);
  if (!load_) return;
  GBC_CUDA(cudaEventRecord(ev_, copy_));
  GBC_CUDA(cudaStreamWaitEvent(work_, ev_, 0));
}

void HostResult::send(size_t q) {
  ready();
  GBC_CUDA(cudaEventRecord(ev_, work_));
  GBC_CUDA(cudaStreamWaitEvent(copy_, ev_, 0));
  GBC_CUDA(cudaMemcpyAsync(items_[q].host, items_[q].dev, items_[q].bytes, cudaMemcpyDeviceToHost, copy_));
}

void HostResult::wait() { GBC_CUDA(cudaStreamSynchronize(copy_)); }

}  // namespace gbc
