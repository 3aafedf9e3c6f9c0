// host_buffers.hpp -- the caller's result arrays on the host.
//
// A fresh host array has no pages yet.  A device-to-host copy makes them one
// after the other: on the GB300 host a copy into fresh memory runs at 25 GB/s,
// into memory with pages at 190.  populate() makes the pages first, with
// several threads (529 MB: 19.1 ms for the copy alone, 9.2 ms for populate and
// copy; 33 MB: 1.34 against 0.70 ms; more than four threads are slower), or
// while the GPU still computes.
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cstddef>
#include <cstdint>
#include <exception>
#include <thread>
#include <vector>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace lbm {

// Gives [p, p + n) its pages, contents unchanged, if it is ordinary host
// memory of at least a megabyte that has none yet (a few pages are looked at).
// Where the kernel cannot, the copy makes them as it did before.
inline void populate(void* p, size_t n) {
  if (!p || n < ((size_t)1 << 20)) return;
  const long ps = sysconf(_SC_PAGESIZE);
  if (ps <= 0) return;
  const uintptr_t page = (uintptr_t)ps, first = ((uintptr_t)p + page - 1) / page * page,
                  end = ((uintptr_t)p + n) / page * page;
  if (end <= first) return;
  const uintptr_t pages = (end - first) / page;
  int present = 0;
  constexpr int kLook = 3;
  for (int k = 0; k < kLook; ++k) {
    unsigned char in = 0;
    const uintptr_t at_page = first + (pages - 1) * k / (kLook - 1) * page;
    if (mincore((void*)at_page, page, &in) != 0) return;
    present += in & 1;
  }
  if (present == kLook) return;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (at.type != cudaMemoryTypeUnregistered) return;   // pinned, managed: pages are there
  auto make = [=](uintptr_t from, uintptr_t to) {
    if (to > from) (void)madvise((void*)from, to - from, MADV_POPULATE_WRITE);
  };
  const int threads = n < ((size_t)8 << 20) ? 1 : 4;
  const uintptr_t part = (pages + threads - 1) / threads * page;
  std::vector<std::thread> t;
  try {
    t.reserve(threads);
    for (int k = 1; k < threads; ++k) {
      const uintptr_t from = first + k * part;
      if (from < end) t.emplace_back(make, from, from + part < end ? from + part : end);
    }
  } catch (const std::exception&) {   // no more threads or memory: the copy makes the other pages
  }
  make(first, first + part < end ? first + part : end);
  for (std::thread& x : t) x.join();
}

}  // namespace lbm
