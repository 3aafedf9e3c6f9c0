// mapped_result.hpp -- a handle's small results in host memory that the GPU writes.
//
// A kernel writes an objective or a flag straight into host memory, without a
// copy behind it.  Each handle has a page of its own, so nothing is shared
// between handles or threads and nothing outlives the handle.  GB300's GPU
// reads the host's own page tables, so ordinary memory will do; elsewhere the
// page is registered.  (On the GB300 host that takes 25 us, and giving it back
// 20; cudaHostAlloc and cudaFreeHost take 100 and 165.  A single step of a 64x48
// channel with its objective takes 24 us either way.)
#pragma once

#include <cuda_runtime.h>
#include <unistd.h>

#include <cstddef>
#include <cstdlib>
#include <cstring>

namespace lbm {

struct MappedResult {
  static constexpr size_t kBytes = 64;
  double* host = nullptr;   // null until taken
  double* dev = nullptr;    // its device address
  bool registered = false;

  // Takes the page, if there is none yet.  After an error there is none.
  cudaError_t take() {
    if (host) return cudaSuccess;
    const long page = sysconf(_SC_PAGESIZE);
    const size_t n = page > 0 ? (size_t)page : 65536;
    void* p = nullptr;
    if (posix_memalign(&p, n, n) != 0) return cudaErrorMemoryAllocation;
    memset(p, 0, kBytes);
    int device = 0, host_tables = 0;
    void* d = p;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess)
      e = cudaDeviceGetAttribute(&host_tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables,
                                 device);
    if (e == cudaSuccess && !host_tables) {
      e = cudaHostRegister(p, kBytes, cudaHostRegisterMapped | cudaHostRegisterPortable);
      if (e == cudaSuccess && (e = cudaHostGetDevicePointer(&d, p, 0)) != cudaSuccess)
        cudaHostUnregister(p);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      free(p);
      return e;
    }
    host = (double*)p;
    dev = (double*)d;
    registered = !host_tables;
    return cudaSuccess;
  }
  // Gives it back; the work that writes to it has ended.
  void give() {
    if (!host) return;
    if (registered && cudaHostUnregister(host) != cudaSuccess) cudaGetLastError();
    free(host);
    host = dev = nullptr;
    registered = false;
  }
};

}  // namespace lbm
