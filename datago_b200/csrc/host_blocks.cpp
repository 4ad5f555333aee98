#include "host_blocks.h"

#include <cuda_runtime.h>
#include <pthread.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <unordered_map>
#include <utility>
#include <vector>

#include "../../include/datago_b200.h"
#include "host.h"

namespace dg {

namespace {

struct Pool {
    std::mutex mu;
    struct Entry { size_t size; int refs; };
    std::unordered_map<void*, Entry> blocks;
    std::multimap<size_t, void*> free;  // those with refs == 0, by size
    std::map<int, int> contexts;  // live ones per device
    int last_device = -1;
    size_t busy = 0, idle = 0, limit;
    size_t peak = 0;  // most that was referenced at one time while there were feeders
    int feeders = 0;
    void add_busy(size_t n) {
        busy += n;
        if (feeders > 0 && busy > peak) peak = busy;
    }
    // idle bytes to keep
    size_t keep() const { return contexts.empty() ? 0 : peak > busy + limit ? peak - busy : limit; }
    Pool() {
        const char* mb = getenv("DATAGO_B200_HOST_BLOCKS_MB");
        const long v = mb ? atol(mb) : 1024;
        limit = (size_t)(v >= 0 ? v : 1024) << 20;
    }
    // takes idle blocks out of the pool while it holds more than `most` bytes of them; the caller unlocks and frees them
    void trim(size_t most, std::vector<std::pair<void*, size_t>>* gone) {
        while (!free.empty() && idle > most) {
            const auto it = free.begin();
            idle -= it->first;
            gone->emplace_back(it->second, it->first);
            blocks.erase(it->second);
            free.erase(it);
        }
    }
    int device() const { return contexts.empty() ? last_device : contexts.count(last_device) ? last_device : contexts.begin()->first; }
};

Pool& pool() {
    static Pool* p = [] {
        static Pool* made = new Pool();  // deliberately leaked: arrays may outlive static destructors
        // no other thread is in the middle of it when a process forks: the child hands its inherited arrays back as well
        pthread_atfork([] { made->mu.lock(); }, [] { made->mu.unlock(); }, [] { made->mu.unlock(); });
        return made;
    }();
    return *p;
}

constexpr size_t kHuge = (size_t)2 << 20;

size_t rounded(size_t n) {  // eight sizes per power of two, so that blocks of similar batches can stand in for one another
    size_t step = (size_t)64 << 10;
    while (step * 16 <= n) step *= 2;
    return (n + step - 1) / step * step;
}

// Runs f with `device` current and leaves the calling thread as it is: making another device current, or going back to one
// that was never used, creates a context there, so a thread of its own does it.  False: no thread to be had, f has not run.
template <class F>
bool on_device(int device, F&& f) {
    int now = -1;
    if (device < 0 || (cudaGetDevice(&now) == cudaSuccess && now == device)) { f(); return true; }
    try {
        std::thread([&] { cudaSetDevice(device); f(); }).join();
    } catch (const std::system_error&) {
        return false;
    }
    return true;
}

void* map_block(size_t size) {
    const size_t extra = size >= kHuge ? kHuge : 0;  // large blocks start at a huge page: locking them is four times as quick
    void* at = mmap(nullptr, size + extra, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (at == MAP_FAILED) return nullptr;
    if (!extra) return at;
    uint8_t* const a = (uint8_t*)at;
    uint8_t* const p = (uint8_t*)(((uintptr_t)a + kHuge - 1) / kHuge * kHuge);
    if (p != a) munmap(a, (size_t)(p - a));
    if (p + size != a + size + extra) munmap(p + size, (size_t)(a + size + extra - (p + size)));
    madvise(p, size, MADV_HUGEPAGE);
    return p;
}

void free_all(const std::vector<std::pair<void*, size_t>>& gone, int device) {
    if (gone.empty()) return;
    const auto unlock = [&] {
        for (const auto& b : gone) cudaHostUnregister(b.first);
        cudaGetLastError();
    };
    if (!on_device(device, unlock)) unlock();
    for (const auto& b : gone) munmap(b.first, b.second);
}

int acquire(size_t nbytes, bool optional, void** out) {
    Pool& p = pool();
    const size_t need = rounded(nbytes ? nbytes : 1);
    int device;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if (optional && p.busy + need > p.limit) return dg_set_error(DG_E_TOO_LARGE, "host blocks: too much is in use");
        const auto it = p.free.lower_bound(need);
        if (it != p.free.end() && it->first <= 2 * need) {
            *out = it->second;
            madvise(it->second, it->first, MADV_DOFORK);
            p.idle -= it->first;
            p.add_busy(it->first);
            p.blocks[it->second].refs = 1;
            p.free.erase(it);
            return DG_OK;
        }
        p.add_busy(need);
        device = p.device();
    }
    void* const ptr = map_block(need);
    cudaError_t err = cudaErrorMemoryAllocation;
    if (ptr) on_device(device, [&] { if ((err = cudaHostRegister(ptr, need, cudaHostRegisterPortable)) != cudaSuccess) cudaGetLastError(); });
    std::lock_guard<std::mutex> lock(p.mu);
    if (err != cudaSuccess) {
        if (ptr) munmap(ptr, need);
        p.busy -= need;
        return dg_set_error(DG_E_CUDA, "host blocks: page-locked allocation failed");
    }
    p.blocks.emplace(ptr, Pool::Entry{need, 1});
    *out = ptr;
    return DG_OK;
}

}  // namespace

int host_block_acquire(size_t nbytes, bool optional, void** out) {
    *out = nullptr;
    try {
        return acquire(nbytes, optional, out);
    } catch (const std::bad_alloc&) {
        return dg_set_error(DG_E_CUDA, "host blocks: out of memory");
    }
}

void host_block_retain(void* base) {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    auto it = p.blocks.find(base);
    if (it != p.blocks.end()) ++it->second.refs;
}

void host_block_release(void* base) {
    if (!base) return;
    Pool& p = pool();
    std::vector<std::pair<void*, size_t>> gone;
    int device;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        auto it = p.blocks.find(base);
        if (it == p.blocks.end() || it->second.refs == 0) return;
        if (--it->second.refs) return;
        p.busy -= it->second.size;
        p.idle += it->second.size;
        madvise(base, it->second.size, MADV_DONTFORK);
        p.free.emplace(it->second.size, base);
        p.trim(p.keep(), &gone);
        device = p.device();
    }
    free_all(gone, device);
}

bool host_blocks_scarce() {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    return p.busy > p.limit;
}

bool host_blocks_room(size_t nbytes) {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    return p.busy + nbytes <= p.limit;
}

void host_blocks_context(int device, int change) {
    Pool& p = pool();
    std::vector<std::pair<void*, size_t>> gone;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if ((p.contexts[device] += change) <= 0) p.contexts.erase(device);
        p.last_device = device;
        p.trim(p.keep(), &gone);
    }
    free_all(gone, device);
}

void host_blocks_feeder(int change) {
    Pool& p = pool();
    std::vector<std::pair<void*, size_t>> gone;
    int device;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        p.feeders += change;
        if (p.feeders <= 0) p.peak = 0;
        p.trim(p.keep(), &gone);
        device = p.device();
    }
    free_all(gone, device);
}

}  // namespace dg

extern "C" int dg_host_alloc(uint64_t nbytes, void** out) {
    if (!out) return dg::dg_set_error(DG_E_INVALID, "out is NULL");
    return dg::host_block_acquire((size_t)nbytes, true, out);
}
extern "C" void dg_host_release(void* block) { dg::host_block_release(block); }
