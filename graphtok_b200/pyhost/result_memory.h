// Memory of large results.
//
// A fresh array of megabytes pays for its pages as it is filled: encoding a 4.5 MB document takes 785 us into fresh memory (huge
// pages) and 405 into memory that was used before, a 32 MB corpus file (56 MB of ids) 7.4 ms and 3.7.  Programs that encode file
// after file drop one result before or soon after they ask for the next, so the memory of dropped results is kept for the ones
// to come, bounded, while a tokenizer is open.  It is ordinary
// memory that the array owns, from malloc: an asynchronous copy from it is staged before the copy's call returns, a forked
// child has its own copy, and ndarray.resize works, none of which holds for page-locked blocks that are handed out again.
#pragma once
#include <malloc.h>
#include <sys/mman.h>

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <mutex>

namespace result_memory {

constexpr size_t kLeast = 256 << 10;         // results below it are malloc's alone: it has such sizes at hand itself
constexpr size_t kHuge = 4 << 20;            // huge pages are asked for from here on, as numpy does
// What is kept at most: two threads with two results each, of the longest texts that are usual in one call.
constexpr int kMostKept = 4;
constexpr size_t kMostBytes = 256 << 20;

struct Kept {
    std::mutex mu;
    void* at[kMostKept];
    size_t size[kMostKept];                  // oldest first
    int n = 0;
    size_t bytes = 0;
    int users = 0;

    void* take(int i) {
        void* p = at[i];
        bytes -= size[i];
        for (--n; i < n; ++i) { at[i] = at[i + 1]; size[i] = size[i + 1]; }
        return p;
    }
};
inline Kept& kept() {
    static Kept* k = new Kept();             // never destroyed: arrays may be dropped while the process ends
    return *k;
}

inline void* get(size_t bytes) {
    // an eighth to spare, so that results of about the same size fit each other's memory (it costs nothing until it is used)
    const size_t want = (bytes + bytes / 8 + 4095) & ~size_t(4095);
    Kept& k = kept();
    {
        std::unique_lock<std::mutex> lock(k.mu, std::try_to_lock);      // (never waits: a fork may have left it locked)
        int best = -1;
        if (lock.owns_lock())
            for (int i = 0; i < k.n; ++i)
                if (k.size[i] >= bytes && k.size[i] / 2 <= want && (best < 0 || k.size[i] < k.size[best])) best = i;
        if (best >= 0) return k.take(best);
    }
    void* p = std::malloc(want);
    if (p && want >= kHuge) {
        const uintptr_t page = (reinterpret_cast<uintptr_t>(p) + 4095) & ~uintptr_t(4095);
        madvise(reinterpret_cast<void*>(page), want - (page - reinterpret_cast<uintptr_t>(p)), MADV_HUGEPAGE);
    }
    return p;
}

inline void put(void* p) {
    const size_t size = p ? malloc_usable_size(p) : 0;
    if (size >= kLeast && size <= kMostBytes) {
        Kept& k = kept();
        std::unique_lock<std::mutex> lock(k.mu, std::try_to_lock);
        if (lock.owns_lock() && k.users > 0) {
            while (k.n == kMostKept || k.bytes + size > kMostBytes) std::free(k.take(0));
            k.at[k.n] = p;
            k.size[k.n++] = size;
            k.bytes += size;
            return;
        }
    }
    std::free(p);
}

// +1 for each tokenizer that is opened, -1 when it is closed: with the last one what is kept goes back to the system.
inline void users(int change) {
    Kept& k = kept();
    std::lock_guard<std::mutex> lock(k.mu);
    k.users += change;
    while (k.users <= 0 && k.n) std::free(k.take(0));
}

}  // namespace result_memory
