// See result_blocks.h.
#include "result_blocks.h"

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace gtok {

namespace {

// Both bounds count free blocks and blocks in use.  Six blocks are what three threads with two results each
// hold; 1 GiB is two results of the longest texts that are worth one call.
constexpr size_t kMostBlocks = 6;
constexpr size_t kMostBytes = size_t(1) << 30;

struct Block {
    void* p;
    size_t bytes;
    bool used;
};
struct Pool {
    std::mutex mu;
    std::vector<Block> blocks;
    size_t bytes = 0;
    int users = 0;
};
// Never destroyed: blocks may be given back while the process ends, after static objects are gone.
Pool& pool() {
    static Pool* p = new Pool();
    return *p;
}

void drop(Pool& pl, size_t i) {
    if (cudaFreeHost(pl.blocks[i].p) != cudaSuccess) cudaGetLastError();
    pl.bytes -= pl.blocks[i].bytes;
    pl.blocks.erase(pl.blocks.begin() + static_cast<std::ptrdiff_t>(i));
}

}  // namespace

void* result_block_get(size_t bytes) {
    Pool& pl = pool();
    std::lock_guard<std::mutex> lock(pl.mu);
    const size_t none = ~size_t(0);
    size_t best = none;
    for (size_t i = 0; i < pl.blocks.size(); ++i)
        if (!pl.blocks[i].used && pl.blocks[i].bytes >= bytes && (best == none || pl.blocks[i].bytes < pl.blocks[best].bytes)) best = i;
    const size_t want = (bytes + bytes / 4 + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);
    const bool room = pl.blocks.size() < kMostBlocks && pl.bytes + want <= kMostBytes;
    // (a block many times the size is only taken where there is no room for one of the right size)
    if (best != none && (pl.blocks[best].bytes <= 4 * want || !room)) {
        pl.blocks[best].used = true;
        return pl.blocks[best].p;
    }
    // none that is free will do: a new one with a quarter to spare, in place of the smallest free ones where the bounds ask for it
    while (pl.blocks.size() >= kMostBlocks || pl.bytes + want > kMostBytes) {
        size_t victim = none;
        for (size_t i = 0; i < pl.blocks.size(); ++i)
            if (!pl.blocks[i].used && (victim == none || pl.blocks[i].bytes < pl.blocks[victim].bytes)) victim = i;
        if (victim == none) return nullptr;
        drop(pl, victim);
    }
    void* p = nullptr;
    if (cudaHostAlloc(&p, want, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    pl.blocks.push_back({p, want, true});
    pl.bytes += want;
    return p;
}

void result_block_put(void* block) {
    Pool& pl = pool();
    std::lock_guard<std::mutex> lock(pl.mu);
    for (size_t i = 0; i < pl.blocks.size(); ++i)
        if (pl.blocks[i].p == block) {
            pl.blocks[i].used = false;
            if (pl.users == 0) drop(pl, i);
            return;
        }
}

void result_blocks_user(int change) {
    Pool& pl = pool();
    std::lock_guard<std::mutex> lock(pl.mu);
    pl.users += change;
    if (pl.users > 0) return;
    for (size_t i = pl.blocks.size(); i-- > 0;)
        if (!pl.blocks[i].used) drop(pl, i);
}

}  // namespace gtok
