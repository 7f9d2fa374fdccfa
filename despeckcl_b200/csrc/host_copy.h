// Copies between pageable host memory and the device through pinned slots,
// the host side on several threads.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace dcl {

// Slots of a call, and a slot's size: 1531 x 1999 takes 10.1 ms with 8 and with
// 4 MiB, 10.9 with 2; 3000 x 3000 28.2, 28.9 and 33.1 ms.  A block of 16 MiB
// takes about 7 ms to pin, once.
constexpr int kSlots = 4;
constexpr size_t kSlotBytes = size_t(4) << 20;

// The pinned slots of one host-pointer call, used for its uploads, then for its
// downloads.  A block of them is pinned when none is idle (that takes longer
// than the copies it serves), then serves later calls of any thread: a program
// that starts a thread per scene would pay for it on every call otherwise (1000
// x 1000 took 37.7 ms a call with slots of the thread's own, 3.9 ms now; 4.7
// without slots).  At
// most kMaxBlocks are pinned at a time; those that no kWindow calls in a row
// needed at once are given back, down to one.
class PinnedBlock {
 public:
  static constexpr int kMaxBlocks = 4, kWindow = 64;
  static constexpr size_t kBytes = kSlots * kSlotBytes;
  PinnedBlock() = default;
  ~PinnedBlock();  // the call's copies have ended
  PinnedBlock(const PinnedBlock&) = delete;
  PinnedBlock& operator=(const PinnedBlock&) = delete;
  // false where all blocks are in use or no more can be pinned now
  bool take();
  char* slot(size_t i) const { return mem_ + i % kSlots * kSlotBytes; }
  // calls that held a block when this one took its own, itself included
  int sharers() const { return sharers_; }

 private:
  char* mem_ = nullptr;
  int sharers_ = 0;
};

// When the copies of a thread's slots have ended, per device.
struct SlotEvents {
  cudaEvent_t ev[kSlots] = {};
  // false where the events cannot be had now
  bool ready();
  cudaEvent_t at(size_t i) const { return ev[i % kSlots]; }
  ~SlotEvents();
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
