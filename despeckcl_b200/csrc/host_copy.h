// Copies between pageable host memory and the device through pinned slots,
// the host side on several threads.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace dcl {

// Pinned slots of a thread's host-pointer calls, made on first use and given
// back when the thread ends.
struct PinnedSlots {
  static constexpr int kSlots = 4;
  static constexpr size_t kSlotBytes = size_t(8) << 20;
  char* mem = nullptr;
  cudaEvent_t ev[kSlots] = {};
  bool ok = false, tried = false;
  // false where the memory or the events cannot be had
  bool ready();
  char* slot(int i) const { return mem + (size_t)(i % kSlots) * kSlotBytes; }
  ~PinnedSlots();
};

// Threads that live for one call and copy together with the caller.
class CopyCrew {
 public:
  explicit CopyCrew(int threads);
  ~CopyCrew();
  CopyCrew(const CopyCrew&) = delete;
  CopyCrew& operator=(const CopyCrew&) = delete;
  // memcpy, split over the crew; returns when done
  void copy(void* dst, const void* src, size_t bytes);

 private:
  struct Impl;
  Impl* impl_;
};

// Whether `p` is pageable memory (not pinned, managed or device memory).
bool is_pageable(const void* p);

}  // namespace dcl
