"""csrc/host_copy.cpp on the CPU, linked against a stand-in for the few CUDA calls
it makes: blocks of pinned memory serve later calls of any thread, stay within
their bound, are given back when they are no longer needed at once, and a call
that could not get one leaves nothing behind; the crew copies every byte."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "despeckcl_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <thread>
#include <vector>
#include "host_copy.h"
using namespace dcl;

static std::atomic<int> allocs{0}, frees{0}, events{0}, fail_alloc{0}, fail_event{0};
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (fail_alloc > 0) return --fail_alloc, cudaErrorMemoryAllocation;
  ++allocs;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { ++frees; std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (fail_event > 0 && --fail_event == 0) return cudaErrorMemoryAllocation;
  ++events;
  *e = (cudaEvent_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { --events; std::free((void*)e); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
}
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
  // a thread per call, one after another: pinned once
  for (int i = 0; i < 20; ++i)
    std::thread([] { PinnedBlock b; if (!b.take()) std::abort(); std::memset(b.slot(3), 1, kSlotBytes); }).join();
  CHECK(allocs == 1 && frees == 0);
  // the first allocation to fail is tried again by the next call
  {
    PinnedBlock a, b, c;
    CHECK(a.take());
    fail_alloc = 1;
    CHECK(!b.take());
    CHECK(c.take() && b.take());
    CHECK(a.sharers() == 1 && b.sharers() == 3);
  }
  // a bound on the blocks in use at once
  {
    std::vector<std::unique_ptr<PinnedBlock>> held;
    for (int i = 0; i < PinnedBlock::kMaxBlocks; ++i) {
      held.emplace_back(new PinnedBlock);
      CHECK(held.back()->take() && held.back()->take());
    }
    PinnedBlock more;
    CHECK(!more.take());
    held.pop_back();
    CHECK(more.take());
  }
  CHECK(allocs - frees == PinnedBlock::kMaxBlocks);
  // two windows of calls one at a time: given back, down to one
  for (int i = 0; i < 2 * PinnedBlock::kWindow; ++i) {
    PinnedBlock b;
    CHECK(b.take());
  }
  CHECK(allocs - frees == 1);
  // calls from several threads, each with its own block
  std::atomic<int> bad{0};
  std::vector<std::thread> t;
  for (int k = 0; k < 6; ++k)
    t.emplace_back([&bad, k] {
      for (int i = 0; i < 200; ++i) {
        PinnedBlock b;
        if (!b.take()) continue;
        std::memset(b.slot(i), k, 4096);
        std::this_thread::yield();
        for (int j = 0; j < 4096; ++j) bad += b.slot(i)[j] != k;
      }
    });
  for (auto& x : t) x.join();
  CHECK(bad == 0 && allocs - frees <= PinnedBlock::kMaxBlocks);
  // events that cannot be made are tried again, none is lost
  {
    SlotEvents e;
    fail_event = 3;
    CHECK(!e.ready());
    CHECK(e.ready() && events == kSlots);
  }
  CHECK(events == 0);
  // the crew: sizes around its pieces, many jobs in a row
  for (int threads : {0, 1, 4}) {
    CopyCrew crew(threads);
    for (size_t n : {size_t(1), (size_t(256) << 10) - 1, (size_t(256) << 10) + 1, (size_t(3) << 20) + 17})
      for (int rep = 0; rep < 20; ++rep) {
        std::vector<char> a(n), b(n + 1, 3);
        for (size_t i = 0; i < n; ++i) a[i] = (char)(i * 7 + rep);
        crew.copy(b.data(), a.data(), n);
        CHECK(std::memcmp(a.data(), b.data(), n) == 0 && b[n] == 3);
      }
  }
  std::puts("ok");
  return 0;
}
"""


def test_pinned_blocks_and_copy_crew(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    src = tmp_path / "main.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(CUDA, "include"), str(src),
                    os.path.join(CSRC, "host_copy.cpp"), "-pthread", "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.stdout.strip() == "ok" and out.returncode == 0, out.stdout + out.stderr
