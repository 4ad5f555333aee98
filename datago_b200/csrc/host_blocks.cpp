#include "host_blocks.h"

#include <cuda_runtime.h>

#include <cstdlib>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "../../include/datago_b200.h"
#include "host.h"

namespace dg {

namespace {

struct Pool {
    std::mutex mu;
    struct Entry { size_t size; int refs; };
    std::unordered_map<void*, Entry> blocks;
    size_t busy = 0, idle = 0, limit;
    int contexts = 0;
    Pool() {
        const char* mb = getenv("DATAGO_B200_HOST_BLOCKS_MB");
        const long v = mb ? atol(mb) : 1024;
        limit = (size_t)(v >= 0 ? v : 1024) << 20;
    }
    // takes the idle blocks out of the pool while it holds more than `most` bytes of them; the caller frees them unlocked
    void trim(size_t most, std::vector<void*>* gone) {
        for (auto it = blocks.begin(); it != blocks.end() && idle > most;) {
            if (it->second.refs == 0) {
                idle -= it->second.size;
                gone->push_back(it->first);
                it = blocks.erase(it);
            } else ++it;
        }
    }
};

Pool& pool() {
    static Pool* p = new Pool();  // deliberately leaked: arrays may outlive static destructors
    return *p;
}

size_t rounded(size_t n) {  // eight sizes per power of two, so that blocks of similar batches can stand in for one another
    size_t step = (size_t)64 << 10;
    while (step * 16 <= n) step *= 2;
    return (n + step - 1) / step * step;
}

void free_all(const std::vector<void*>& gone) {
    for (void* p : gone) cudaFreeHost(p);
}

}  // namespace

int host_block_acquire(size_t nbytes, bool optional, void** out) {
    Pool& p = pool();
    const size_t need = rounded(nbytes ? nbytes : 1);
    *out = nullptr;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if (optional && p.busy + need > p.limit) return dg_set_error(DG_E_TOO_LARGE, "host blocks: too much is in use");
        void* best = nullptr;
        for (auto& e : p.blocks)
            if (e.second.refs == 0 && e.second.size >= need && e.second.size <= 2 * need && (!best || e.second.size < p.blocks[best].size)) best = e.first;
        if (best) {
            Pool::Entry& e = p.blocks[best];
            e.refs = 1;
            p.idle -= e.size;
            p.busy += e.size;
            *out = best;
            return DG_OK;
        }
        p.busy += need;
    }
    void* ptr = nullptr;
    const cudaError_t err = cudaHostAlloc(&ptr, need, cudaHostAllocPortable);
    std::lock_guard<std::mutex> lock(p.mu);
    if (err != cudaSuccess) {
        cudaGetLastError();
        p.busy -= need;
        return dg_set_error(DG_E_CUDA, "host blocks: page-locked allocation failed");
    }
    p.blocks.emplace(ptr, Pool::Entry{need, 1});
    *out = ptr;
    return DG_OK;
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
    std::vector<void*> gone;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        auto it = p.blocks.find(base);
        if (it == p.blocks.end() || it->second.refs == 0) return;
        if (--it->second.refs) return;
        p.busy -= it->second.size;
        p.idle += it->second.size;
        p.trim(p.contexts > 0 ? p.limit : 0, &gone);
    }
    free_all(gone);
}

bool host_blocks_scarce() {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    return p.busy > p.limit;
}

void host_blocks_context(int change) {
    Pool& p = pool();
    std::vector<void*> gone;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        p.contexts += change;
        if (p.contexts <= 0) p.trim(0, &gone);
    }
    free_all(gone);
}

}  // namespace dg

extern "C" int dg_host_alloc(uint64_t nbytes, void** out) {
    if (!out) return dg::dg_set_error(DG_E_INVALID, "out is NULL");
    return dg::host_block_acquire((size_t)nbytes, true, out);
}
extern "C" void dg_host_release(void* block) { dg::host_block_release(block); }
