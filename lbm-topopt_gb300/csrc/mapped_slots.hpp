// mapped_slots.hpp -- small results in mapped host memory, one slot per handle.
//
// A kernel writes an objective or a flag straight into host memory, without a
// copy behind it.  Allocating and freeing that memory costs some 100 and 170 us,
// more than everything else of a small handle's creation, so handles share
// pages of 64 slots.  One page is kept when the last handle is gone; further
// ones are given back as soon as they are empty.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <new>

namespace lbm {

class MappedSlots {
 public:
  static constexpr size_t kSlot = 64;   // bytes
  // A free slot, or null (with CUDA's error).
  static void* take(cudaError_t* err) {
    std::lock_guard<std::mutex> lock(mutex());
    Page*& head = pages();
    Page* p = head;
    while (p && p->used == ~0ull) p = p->next;
    if (!p) {
      void* mem = nullptr;
      *err = cudaHostAlloc(&mem, 64 * kSlot, cudaHostAllocMapped | cudaHostAllocPortable);
      if (*err != cudaSuccess) return nullptr;
      p = new (std::nothrow) Page;
      if (!p) {
        cudaFreeHost(mem);
        *err = cudaErrorMemoryAllocation;
        return nullptr;
      }
      p->mem = (char*)mem;
      p->next = head;
      head = p;
    }
    int k = 0;
    while (p->used >> k & 1ull) ++k;
    p->used |= 1ull << k;
    *err = cudaSuccess;
    return p->mem + k * kSlot;
  }
  static void give(void* slot) {
    std::lock_guard<std::mutex> lock(mutex());
    for (Page** at = &pages(); *at; at = &(*at)->next) {
      Page* p = *at;
      const uintptr_t off = (uintptr_t)slot - (uintptr_t)p->mem;
      if ((uintptr_t)slot < (uintptr_t)p->mem || off >= 64 * kSlot) continue;
      p->used &= ~(1ull << (off / kSlot));
      if (p->used == 0ull && (p != pages() || p->next)) {   // not the only page
        *at = p->next;
        cudaFreeHost(p->mem);
        delete p;
      }
      return;
    }
  }

 private:
  struct Page {
    char* mem = nullptr;
    uint64_t used = 0;
    Page* next = nullptr;
  };
  static std::mutex& mutex() {
    static std::mutex m;
    return m;
  }
  static Page*& pages() {
    static Page* head = nullptr;
    return head;
  }
};

}  // namespace lbm
