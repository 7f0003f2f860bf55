// Copies between the device and a caller's host memory in pieces.
//
// A fresh host array has no pages yet, and a device-to-host copy then faults
// them in one after another on one thread: 29 ms for 759 MB that the copy
// itself takes 4 ms for.  PageTouch faults the destination's pages in on a few
// threads, piece by piece ahead of the copy: 8 threads reach 130 GB/s where
// one reaches 27 (64 KB pages, 16 cores; madvise(MADV_POPULATE_WRITE) stays
// at 35 whatever the threads).
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <memory>
#include <thread>
#include <vector>

namespace umwm {

// Bytes per piece: the staging buffer of a transposed copy, small enough to
// stay in L2 between the transpose and the copy.  759 MB to pinned memory take
// 4.5 ms in pieces of 32 MB, 4.6 of 16 and 5.3 of 8 (3.9 as one copy of what
// is there already); to fresh pages 9.4 ms.
constexpr size_t COPY_PIECE = (size_t)32 << 20;

class PageTouch {
 public:
  // Pages of [p, p + bytes), in pieces of `piece` bytes; nothing to do for
  // memory that is pinned, managed or the device's, for a small copy, or where
  // the pages are there (an array that the caller keeps: starting the threads
  // took longer than it saved, 51 MB 0.64 ms against 0.43 without).
  PageTouch(void* p, size_t bytes, size_t piece) : p_(static_cast<char*>(p)), bytes_(bytes), piece_(piece) {
    if (bytes < MIN_BYTES || piece == 0) return;
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    if (at.type != cudaMemoryTypeUnregistered || !fresh()) return;
    const size_t cores = std::max(1u, std::thread::hardware_concurrency());
    const size_t nt = std::min({(size_t)8, std::max<size_t>(cores / 2, 1), bytes / MIN_BYTES});
    try {
      done_.reset(new std::atomic<int>[nt]);
      for (size_t t = 0; t < nt; ++t) done_[t].store(0, std::memory_order_relaxed);
      th_.reserve(nt);
      for (size_t t = 0; t < nt; ++t) th_.emplace_back([this, t, nt] { work(t, nt); });
    } catch (...) {  // no thread or memory left: the copy faults the rest in itself
    }
  }
  ~PageTouch() {
    for (std::thread& t : th_) t.join();
  }
  PageTouch(const PageTouch&) = delete;
  PageTouch& operator=(const PageTouch&) = delete;

  // until piece c's pages are there
  void wait(size_t c) const {
    for (size_t t = 0; t < th_.size(); ++t)
      while ((size_t)done_[t].load(std::memory_order_acquire) <= c) std::this_thread::yield();
  }

 private:
  static constexpr size_t MIN_BYTES = (size_t)4 << 20;

  // whether MIN_BYTES or more of the range has no page yet (or the kernel does not say)
  bool fresh() const {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const uintptr_t base = reinterpret_cast<uintptr_t>(p_);
    unsigned char there[1024];
    size_t missing = 0;
    for (uintptr_t a = (base + page - 1) / page * page; a < base + bytes_; a += sizeof there * page) {
      const size_t n = std::min(sizeof there, (base + bytes_ - a + page - 1) / page);
      if (mincore(reinterpret_cast<void*>(a), n * page, there) != 0) return true;
      for (size_t i = 0; i < n; ++i) missing += !(there[i] & 1);
      if (missing * page >= MIN_BYTES) return true;
    }
    return false;
  }
  // thread t's share of each piece: the pages that start in it.  A plain store,
  // of a byte that the copy is about to write: a load first (or an atomic or
  // with 0, which faults as a load) would map the zero page and then have every
  // page replaced, 270 ms for the 759 MB above.
  void work(size_t t, size_t nt) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), pieces = (bytes_ + piece_ - 1) / piece_;
    const uintptr_t base = reinterpret_cast<uintptr_t>(p_);
    for (size_t c = 0; c < pieces; ++c) {
      const size_t b = c * piece_, n = std::min(piece_, bytes_ - b);
      const uintptr_t lo = base + b + n * t / nt, hi = base + b + n * (t + 1) / nt;
      for (uintptr_t q = (lo + page - 1) / page * page; q < hi; q += page) {
        *reinterpret_cast<volatile char*>(q) = 0;
      }
      done_[t].store((int)c + 1, std::memory_order_release);
    }
  }

  char* p_;
  size_t bytes_, piece_;
  std::unique_ptr<std::atomic<int>[]> done_;
  std::vector<std::thread> th_;
};

}  // namespace umwm
