// MappedResult (lbm-topopt_gb300/csrc/mapped_result.hpp) over a fake CUDA runtime
// that counts registrations and fails on request.  Prints "ok".
#include <cstdio>
#include <map>

#include "mapped_result.hpp"

static std::map<void*, int> registered;
static int fail_register = 0, fail_pointer = 0, fail_attribute = 0, host_tables = 0, last_error = 0;

extern "C" {
cudaError_t cudaHostRegister(void* p, size_t, unsigned) {
  if (fail_register) return (cudaError_t)(last_error = cudaErrorMemoryAllocation);
  if (registered.count(p)) return (cudaError_t)(last_error = cudaErrorHostMemoryAlreadyRegistered);
  registered[p] = 1;
  return cudaSuccess;
}
cudaError_t cudaHostUnregister(void* p) {
  if (!registered.erase(p)) return (cudaError_t)(last_error = cudaErrorHostMemoryNotRegistered);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* p, unsigned) {
  if (fail_pointer || !registered.count(p)) return (cudaError_t)(last_error = cudaErrorInvalidValue);
  *d = p;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  if (fail_attribute || a != cudaDevAttrPageableMemoryAccessUsesHostPageTables)
    return (cudaError_t)(last_error = cudaErrorInvalidValue);
  *v = host_tables;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const int e = last_error;
  last_error = 0;
  return (cudaError_t)e;
}
}

#define CHECK(x)                                   \
  do {                                             \
    if (!(x)) {                                    \
      printf("line %d: %s\n", __LINE__, #x);       \
      return 1;                                    \
    }                                              \
  } while (0)

int main() {
  using lbm::MappedResult;
  MappedResult a, b;
  // a failed call leaves nothing behind, and the next one starts afresh
  fail_register = 1;
  CHECK(a.take() != cudaSuccess && !a.host && !a.dev && registered.empty() && last_error == 0);
  fail_register = 0;
  fail_pointer = 1;
  CHECK(a.take() != cudaSuccess && !a.host && !a.dev && registered.empty() && last_error == 0);
  fail_pointer = 0;
  fail_attribute = 1;
  CHECK(a.take() != cudaSuccess && !a.host && !a.dev && registered.empty() && last_error == 0);
  fail_attribute = 0;
  CHECK(a.take() == cudaSuccess && a.host && a.dev == a.host && registered.size() == 1);
  double* const first = a.host;
  CHECK(a.take() == cudaSuccess && a.host == first && registered.size() == 1);
  // every handle has its own; nothing is left when the last is gone
  CHECK(b.take() == cudaSuccess && b.host != a.host && registered.size() == 2);
  b.give();
  b.give();
  CHECK(!b.host && !b.dev && registered.size() == 1);
  a.give();
  CHECK(registered.empty() && last_error == 0);
  // a device reset between two handles, and under a live one
  CHECK(a.take() == cudaSuccess);
  registered.clear();
  a.give();
  CHECK(!a.host && last_error == 0);
  CHECK(a.take() == cudaSuccess && a.dev && registered.size() == 1);
  a.give();
  // a GPU that reads the host's page tables takes the page as it is
  host_tables = 1;
  CHECK(a.take() == cudaSuccess && b.take() == cudaSuccess && registered.empty());
  CHECK(a.host && a.dev == a.host && b.dev == b.host && a.host != b.host);
  *a.host = 3.;
  a.give();
  host_tables = 0;
  CHECK(a.take() == cudaSuccess && registered.size() == 1);
  a.give();
  b.give();
  CHECK(!a.host && !b.host && registered.empty() && last_error == 0);
  printf("ok\n");
  return 0;
}
