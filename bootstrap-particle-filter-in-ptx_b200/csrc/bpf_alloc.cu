// bpf_alloc.cu — allocation wrappers with live-allocation tracking and a one-shot
// injected failure (see bpf_alloc.cuh). The injected failure returns
// cudaErrorMemoryAllocation without calling the runtime, as a real out-of-memory
// allocation would, so callers take their ordinary error path.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "bpf_alloc.cuh"
#include "../../include/gpu_bpf.h"

namespace {
std::mutex g_mutex;
std::unordered_map<void*, size_t> g_live;   // live device and pinned allocations and their bytes
long long g_fail_in = -1;                 // allocations to let through before the injected failure
long long g_count = 0;                    // allocations attempted since load

// true when this allocation is the one to fail
bool take_failure() {
  std::lock_guard<std::mutex> lock(g_mutex);
  ++g_count;
  if (g_fail_in < 0) return false;
  if (g_fail_in == 0) { g_fail_in = -1; return true; }
  --g_fail_in;
  return false;
}

cudaError_t track(cudaError_t e, void** p, size_t bytes) {
  if (e == cudaSuccess && *p) {
    std::lock_guard<std::mutex> lock(g_mutex);
    g_live[*p] = bytes;
  }
  return e;
}

void untrack(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lock(g_mutex);
  g_live.erase(p);
}

// Recursive: an owner's give_back frees under the lock that its caller holds.
std::recursive_mutex g_kept_mutex;
std::vector<KeptOwner*> g_kept;

size_t kept_on(int device) {                // device < 0: on all
  size_t n = 0;
  for (const KeptOwner* o : g_kept) if (device < 0 || o->device == device) n += o->bytes;
  return n;
}

// Every idle owner on the device (all devices if negative) gives its memory back; the bytes given.
size_t kept_trim(int device) {
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  const size_t before = kept_on(device);
  for (KeptOwner* o : g_kept)
    if ((device < 0 || o->device == device) && o->in_use == 0 && o->bytes > 0) o->give_back();
  return before - kept_on(device);
}
}  // namespace

void kept_register(KeptOwner* o) {
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  g_kept.push_back(o);
}
void kept_unregister(KeptOwner* o) {
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  g_kept.erase(std::remove(g_kept.begin(), g_kept.end(), o), g_kept.end());
}
KeptUse::KeptUse(KeptOwner* o) : owner(o) {
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  ++o->in_use;
}
KeptUse::~KeptUse() {
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  --owner->in_use;
}
void kept_malloc(KeptOwner* o, void** p, size_t bytes) {
  *p = nullptr;
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  size_t free_b = 0, total_b = 0;
  const size_t held = kept_on(o->device);
  const bool fits = cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && held + bytes <= (free_b + held) / 8;
  if (!fits || take_failure() || track(cudaMalloc(p, bytes), p, bytes) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return;
  }
  o->bytes += bytes;
}
void kept_free(KeptOwner* o, void* p, size_t bytes) {
  if (!p) return;
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  bpf_free(p);
  o->bytes -= bytes;
}

cudaError_t bpf_malloc_raw(void** p, size_t bytes) {
  if (take_failure()) { *p = nullptr; return cudaErrorMemoryAllocation; }
  cudaError_t e = cudaMalloc(p, bytes);
  int device = 0;
  if (e == cudaErrorMemoryAllocation && cudaGetDevice(&device) == cudaSuccess && kept_trim(device) > 0) {
    cudaGetLastError();
    e = cudaMalloc(p, bytes);
  }
  return track(e, p, bytes);
}
cudaError_t bpf_malloc_host_raw(void** p, size_t bytes) {
  if (take_failure()) { *p = nullptr; return cudaErrorMemoryAllocation; }
  return track(cudaMallocHost(p, bytes), p, bytes);
}
cudaError_t bpf_host_alloc_raw(void** p, size_t bytes, unsigned flags) {
  if (take_failure()) { *p = nullptr; return cudaErrorMemoryAllocation; }
  return track(cudaHostAlloc(p, bytes, flags), p, bytes);
}
cudaError_t bpf_free(void* p) {
  untrack(p);
  return cudaFree(p);
}
cudaError_t bpf_free_host(void* p) {
  untrack(p);
  return cudaFreeHost(p);
}

extern "C" {

int gpu_bpf_debug_fail_alloc(long long k) {
  std::lock_guard<std::mutex> lock(g_mutex);
  g_fail_in = k < 0 ? -1 : k;
  return BPF_OK;
}

long long gpu_bpf_debug_alloc_count(void) {
  std::lock_guard<std::mutex> lock(g_mutex);
  return g_count;
}

long long gpu_bpf_debug_live_allocs(void) {
  std::lock_guard<std::mutex> lock(g_mutex);
  return (long long)g_live.size();
}

size_t gpu_bpf_debug_live_bytes(void) {
  std::lock_guard<std::mutex> lock(g_mutex);
  size_t n = 0;
  for (const auto& a : g_live) n += a.second;
  return n;
}

size_t gpu_bpf_kept_bytes(void) {
  std::lock_guard<std::recursive_mutex> lock(g_kept_mutex);
  return kept_on(-1);
}

size_t gpu_bpf_trim_kept(void) { return kept_trim(-1); }

}  // extern "C"
