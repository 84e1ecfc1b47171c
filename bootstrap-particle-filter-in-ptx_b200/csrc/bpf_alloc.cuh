// bpf_alloc.cuh — every device and pinned allocation the library makes goes through
// these wrappers (except the allocation-free entry point, which makes none). They
// keep the set of live allocations and can be told to fail one allocation on
// purpose (gpu_bpf_debug_fail_alloc), the host-side fault injection with which the
// cleanup of every create path is tested: no GPU fault is involved.
#pragma once
#include <cstddef>
#include <cuda_runtime.h>
#include <functional>

cudaError_t bpf_malloc_raw(void** p, size_t bytes);
cudaError_t bpf_malloc_host_raw(void** p, size_t bytes);
cudaError_t bpf_host_alloc_raw(void** p, size_t bytes, unsigned flags);
cudaError_t bpf_free(void* p);
cudaError_t bpf_free_host(void* p);

template <typename T>
inline cudaError_t bpf_malloc(T** p, size_t bytes) { return bpf_malloc_raw(reinterpret_cast<void**>(p), bytes); }
template <typename T>
inline cudaError_t bpf_malloc_host(T** p, size_t bytes) { return bpf_malloc_host_raw(reinterpret_cast<void**>(p), bytes); }
template <typename T>
inline cudaError_t bpf_host_alloc(T** p, size_t bytes, unsigned flags) {
  return bpf_host_alloc_raw(reinterpret_cast<void**>(p), bytes, flags);
}

// Kept memory: what a gradient run takes only to be faster (every tick's particles, which the backward
// would recompute otherwise). All owners of a device together hold at most an eighth of its memory that
// is free or so held. An owner gives its share back when it goes, when another allocation of the library
// finds the device full, and on gpu_bpf_trim_kept; it then goes on without.
struct KeptOwner {
  int device = 0;
  std::function<void()> give_back;      // waits for the owner's stream and frees with kept_free
  size_t bytes = 0;                     // held (under the registry's lock, as in_use)
  int in_use = 0;                       // host calls that are using the memory: nobody takes it meanwhile
};
void kept_register(KeptOwner* o);
void kept_unregister(KeptOwner* o);     // before the owner goes (waits for a give_back that is under way)
struct KeptUse {                        // a host call that uses the owner's memory
  explicit KeptUse(KeptOwner* o);
  ~KeptUse();
  KeptUse(const KeptUse&) = delete;
  KeptUse& operator=(const KeptUse&) = delete;
  KeptOwner* owner;
};
// Within a KeptUse or give_back, with the owner's device current. kept_malloc: *p stays null beyond the
// bound or where the device is full.
void kept_malloc(KeptOwner* o, void** p, size_t bytes);
void kept_free(KeptOwner* o, void* p, size_t bytes);
