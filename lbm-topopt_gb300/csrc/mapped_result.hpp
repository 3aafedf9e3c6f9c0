// mapped_result.hpp -- a handle's small results in host memory that the GPU maps.
//
// A kernel writes an objective or a flag straight into host memory, without a
// copy behind it.  Each handle has a page of its own, so nothing is shared
// between handles or threads and nothing outlives the handle: 8 us to register
// and 11 us to give back on the GB300 host, where cudaHostAlloc and cudaFreeHost
// take 100 and 165.
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

  // Takes the page, if there is none yet.  After an error there is none.
  cudaError_t take() {
    if (host) return cudaSuccess;
    const long page = sysconf(_SC_PAGESIZE);
    const size_t n = page > 0 ? (size_t)page : 65536;
    void* p = nullptr;
    if (posix_memalign(&p, n, n) != 0) return cudaErrorMemoryAllocation;
    memset(p, 0, kBytes);
    cudaError_t e = cudaHostRegister(p, kBytes, cudaHostRegisterMapped | cudaHostRegisterPortable);
    void* d = nullptr;
    if (e == cudaSuccess && (e = cudaHostGetDevicePointer(&d, p, 0)) != cudaSuccess)
      cudaHostUnregister(p);
    if (e != cudaSuccess) {
      cudaGetLastError();
      free(p);
      return e;
    }
    host = (double*)p;
    dev = (double*)d;
    return cudaSuccess;
  }
  // Gives it back; the work that writes to it has ended.
  void give() {
    if (!host) return;
    if (cudaHostUnregister(host) != cudaSuccess) cudaGetLastError();
    free(host);
    host = dev = nullptr;
  }
};

}  // namespace lbm
