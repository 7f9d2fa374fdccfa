// See host_copy.h.

#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace dcl {

namespace {

// Blocks of the process.  Never destroyed: threads may end after it would be.
struct BlockPool {
  std::mutex mu;
  std::vector<char*> idle;
  int made = 0;              // pinned, idle or in use
  int takes = 0, peak = 0;   // calls of this window, most blocks in use at once in it

  static BlockPool& get() {
    static BlockPool* p = new BlockPool;
    return *p;
  }
};

}  // namespace

bool PinnedBlock::take() {
  if (mem_) return true;
  BlockPool& p = BlockPool::get();
  std::vector<char*> drop;
  bool make = false;
  {
    std::lock_guard<std::mutex> lk(p.mu);
    p.idle.reserve(kMaxBlocks);  // giving back does not allocate
    if (!p.idle.empty()) {
      mem_ = p.idle.back();
      p.idle.pop_back();
    } else if (p.made < kMaxBlocks) {
      make = true;
      ++p.made;
    }
    sharers_ = p.made - (int)p.idle.size();
    p.peak = std::max(p.peak, sharers_);
    if (++p.takes >= kWindow) {
      while (!p.idle.empty() && p.made > p.peak) {
        drop.push_back(p.idle.back());
        p.idle.pop_back();
        --p.made;
      }
      p.takes = 0;
      p.peak = sharers_;
    }
  }
  for (char* m : drop) cudaFreeHost(m);
  if (!make) return mem_ != nullptr;
  if (cudaHostAlloc(reinterpret_cast<void**>(&mem_), kBytes, cudaHostAllocPortable) == cudaSuccess) return true;
  cudaGetLastError();
  mem_ = nullptr;
  std::lock_guard<std::mutex> lk(p.mu);
  --p.made;
  return false;
}

PinnedBlock::~PinnedBlock() {
  if (!mem_) return;
  BlockPool& p = BlockPool::get();
  std::lock_guard<std::mutex> lk(p.mu);
  p.idle.push_back(mem_);
}

bool SlotEvents::ready() {
  for (cudaEvent_t& e : ev)
    if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      cudaGetLastError();
      e = nullptr;
      return false;
    }
  return true;
}

SlotEvents::~SlotEvents() {
  for (cudaEvent_t e : ev)
    if (e) cudaEventDestroy(e);
}

namespace {
constexpr size_t kPieceBytes = size_t(256) << 10;  // what a thread takes at a time
}

struct CopyCrew::Impl {
  std::vector<std::thread> threads;
  std::mutex mu;
  std::condition_variable wake, done;
  // the job: bytes at dst from src in pieces, taken in order
  char* dst = nullptr;
  const char* src = nullptr;
  size_t bytes = 0;
  std::atomic<size_t> next{0};
  unsigned job = 0;   // jobs posted
  int working = 0;    // threads inside the current job
  bool stop = false;

  void take() {
    for (;;) {
      const size_t at = next.fetch_add(kPieceBytes, std::memory_order_relaxed);
      if (at >= bytes) return;
      std::memcpy(dst + at, src + at, std::min(kPieceBytes, bytes - at));
    }
  }

  void loop() {
    std::unique_lock<std::mutex> lk(mu);
    unsigned seen = 0;
    for (;;) {
      wake.wait(lk, [&] { return stop || job != seen; });
      if (stop) return;
      seen = job;
      ++working;
      lk.unlock();
      take();
      lk.lock();
      if (--working == 0) done.notify_one();
    }
  }
};

CopyCrew::CopyCrew(int threads) : impl_(new Impl()) {
  impl_->threads.reserve(threads);
  for (int i = 0; i < threads; ++i) {
    try {
      impl_->threads.emplace_back([this] { impl_->loop(); });
    } catch (const std::exception&) {
      break;  // the caller copies with those there are
    }
  }
}

CopyCrew::~CopyCrew() {
  {
    std::lock_guard<std::mutex> lk(impl_->mu);
    impl_->stop = true;
  }
  impl_->wake.notify_all();
  for (std::thread& t : impl_->threads) t.join();
  delete impl_;
}

void CopyCrew::copy(void* dst, const void* src, size_t bytes) {
  if (impl_->threads.empty() || bytes <= kPieceBytes) {
    std::memcpy(dst, src, bytes);
    return;
  }
  {
    // a thread that woke late for the job before may still look for a piece
    std::unique_lock<std::mutex> lk(impl_->mu);
    impl_->done.wait(lk, [&] { return impl_->working == 0; });
    impl_->dst = static_cast<char*>(dst);
    impl_->src = static_cast<const char*>(src);
    impl_->bytes = bytes;
    impl_->next.store(0, std::memory_order_relaxed);
    ++impl_->job;
  }
  impl_->wake.notify_all();
  impl_->take();
  // no piece is left: wait for the threads still copying one
  std::unique_lock<std::mutex> lk(impl_->mu);
  impl_->done.wait(lk, [&] { return impl_->working == 0; });
}

bool is_pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace dcl
