// The few CUDA runtime calls that host-side memory management makes, on ordinary memory, for tests without a GPU.  Like the
// real runtime, a call creates a context on the calling thread's current device; fake_contexts() tells where.
#include <cstdlib>
#include <map>
#include <mutex>
#include <set>

#include <cuda_runtime.h>
#include <sys/mman.h>

#include "../datago_b200/csrc/block_cache.h"
#include "../datago_b200/csrc/host.h"
#include "../datago_b200/csrc/host_blocks.h"

namespace {
std::mutex mu;
std::set<int> contexts;
std::map<const void*, std::pair<size_t, int>> locked, allocated;  // page-locked memory with its device; device memory
size_t device_limit = ~(size_t)0;
int allocations = 0, locks = 0;
thread_local int current = 0;
size_t total(const std::map<const void*, std::pair<size_t, int>>& m) {
    size_t n = 0;
    for (auto& e : m) n += e.second.first;
    return n;
}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { std::lock_guard<std::mutex> l(mu); current = d; contexts.insert(d); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostRegister(void* p, size_t n, unsigned int) {
    std::lock_guard<std::mutex> l(mu);
    contexts.insert(current);
    locked[p] = {n, current};
    ++locks;
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void* p) {
    std::lock_guard<std::mutex> l(mu);
    contexts.insert(current);
    return locked.erase(p) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> l(mu);
    *p = nullptr;
    if (total(allocated) + n > device_limit) return cudaErrorMemoryAllocation;
    *p = malloc(1);
    allocated[*p] = {n, current};
    ++allocations;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> l(mu);
    if (allocated.erase(p)) free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) {  // a shared mapping, as the driver makes it
    std::lock_guard<std::mutex> l(mu);
    contexts.insert(current);
    *p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_SHARED | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    locked[*p] = {n, current};
    ++allocations;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::mutex> l(mu);
    contexts.insert(current);
    const auto it = locked.find(p);
    if (it == locked.end()) return cudaErrorInvalidValue;
    munmap(p, it->second.first);
    locked.erase(it);
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "?"; }

int fake_contexts(int device) { std::lock_guard<std::mutex> l(mu); return (int)contexts.count(device); }
int fake_locked_on(const void* p) { std::lock_guard<std::mutex> l(mu); auto it = locked.find(p); return it == locked.end() ? -1 : it->second.second; }
size_t fake_locked_bytes() { std::lock_guard<std::mutex> l(mu); return total(locked); }
size_t fake_device_bytes() { std::lock_guard<std::mutex> l(mu); return total(allocated); }
int fake_locks() { std::lock_guard<std::mutex> l(mu); return locks; }
int fake_allocations() { std::lock_guard<std::mutex> l(mu); return allocations; }
void fake_device_limit(size_t n) { std::lock_guard<std::mutex> l(mu); device_limit = n; }

int hb_acquire(size_t n, int optional, void** out) { return dg::host_block_acquire(n, optional != 0, out); }
void hb_retain(void* p) { dg::host_block_retain(p); }
int hb_scarce() { return dg::host_blocks_scarce(); }
void hb_feeder(int change) { dg::host_blocks_feeder(change); }
void hb_context(int device, int change) { dg::host_blocks_context(device, change); }

void* bc_new() { return new dg::BlockCache(false); }
int bc_acquire(void* c, size_t n) { int i = -1; return ((dg::BlockCache*)c)->acquire(n, &i) ? -1 : i; }
void bc_release(void* c, int i) { ((dg::BlockCache*)c)->release(i); }
void bc_delete(void* c) { ((dg::BlockCache*)c)->clear(); delete (dg::BlockCache*)c; }
}

int dg::dg_set_error(int code, const char*) { return code; }
