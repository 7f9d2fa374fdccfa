// See host_copy.h.

#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace dcl {

bool PinnedSlots::ready() {
  if (tried) return ok;
  tried = true;
  cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&mem), kSlots * kSlotBytes, cudaHostAllocPortable);
  for (int i = 0; i < kSlots && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
  if (e != cudaSuccess) cudaGetLastError();
  ok = e == cudaSuccess;
  return ok;
}

PinnedSlots::~PinnedSlots() {
  for (cudaEvent_t e : ev)
    if (e) cudaEventDestroy(e);
  if (mem) cudaFreeHost(mem);
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
  for (int i = 0; i < threads; ++i) {
    try {
      impl_->threads.emplace_back([this] { impl_->loop(); });
    } catch (const std::system_error&) {
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
