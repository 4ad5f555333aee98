// The blocks of device memory or page-locked memory that a context lends to its batches.
//
// A request takes the smallest idle block that fits.  Where none does, the largest idle one (all of them are too small)
// makes room for the new one.  So a context never holds more blocks than its batches had in hand at one time, whatever
// sizes come by, nor a larger one than the largest request asks for; every allocation replaces a block by a larger one or
// adds one to those in hand, so after a few batches of a kind there are none (and nothing is freed) any more.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <string>
#include <vector>

#include "host.h"

namespace dg {

struct Block {
    void* ptr = nullptr;
    size_t size = 0;
    bool busy = false;
};

struct BlockCache {
    bool pinned;
    std::vector<Block> blocks;
    explicit BlockCache(bool p) : pinned(p) {}
    void give_back(Block& b) {
        if (b.ptr) { if (pinned) cudaFreeHost(b.ptr); else cudaFree(b.ptr); }
        b = Block();
    }
    int acquire(size_t size, int* index) {
        if (size == 0) size = 256;
        int best = -1, victim = -1;
        for (size_t i = 0; i < blocks.size(); ++i) {
            if (blocks[i].busy) continue;
            if (blocks[i].size >= size && (best < 0 || blocks[i].size < blocks[best].size)) best = (int)i;
            if (victim < 0 || blocks[i].size > blocks[victim].size) victim = (int)i;
        }
        if (best < 0) {
            if (victim < 0) { blocks.emplace_back(); victim = (int)blocks.size() - 1; }
            give_back(blocks[victim]);
            Block nb;
            nb.size = size + size / 8 + 4096;
            auto allocate = [&] { return pinned ? cudaHostAlloc(&nb.ptr, nb.size, cudaHostAllocDefault) : cudaMalloc(&nb.ptr, nb.size); };
            cudaError_t e = allocate();
            if (e != cudaSuccess) {  // out of memory: without the other idle blocks, then
                cudaGetLastError();  // a failed allocation must not surface again as the next healthy batch's error
                for (Block& b : blocks) if (!b.busy) give_back(b);
                e = allocate();
            }
            if (e != cudaSuccess) {
                cudaGetLastError();
                return dg_set_error(DG_E_CUDA, (std::string(pinned ? "cudaHostAlloc" : "cudaMalloc") + " of " + std::to_string(nb.size) + " bytes: " + cudaGetErrorString(e)).c_str());
            }
            blocks[victim] = nb;
            best = victim;
        }
        blocks[best].busy = true;
        *index = best;
        return DG_OK;
    }
    void release(int index) { if (index >= 0) blocks[index].busy = false; }
    void clear() {
        for (Block& b : blocks) give_back(b);
        blocks.clear();
    }
};

}  // namespace dg
