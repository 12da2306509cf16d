// hostpool.cpp -- the page-locked result-buffer pool (PinnedPool in
// cof_engine.h).  Buffers are portable pinned allocations, usable from every
// device's stream.  Small results are blocks of size classes cut from shared
// slabs; larger ones are allocations of their own, rounded up so that nearby
// sizes reuse each other: pinning takes about 0.4 ms per MiB, and the pieces of a
// bulge search differ by a few per cent, so that rounded to 2 MiB every piece
// larger than all before it was pinned anew in the middle of the search.
#include <cuda_runtime.h>

#include "cof_engine.h"

namespace cof {

PinnedPool &PinnedPool::get() {
    static PinnedPool pool;  // process lifetime; buffers are released at exit
    return pool;
}

char *PinnedPool::alloc_large(size_t want) {
    char *p = nullptr;
    ++allocs_;
    if (cudaHostAlloc((void **)&p, want, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();  // clear the recorded error of the failed call
        // drop what is kept and try once more
        for (auto &kv : free_) cudaFreeHost(kv.second);
        free_.clear();
        free_bytes_ = 0;
        if (cudaHostAlloc((void **)&p, want, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
    }
    return p;
}

uint64_t PinnedPool::allocations() {
    std::lock_guard<std::mutex> lk(mu_);
    return allocs_;
}

char *PinnedPool::acquire(size_t bytes, size_t at_least, size_t *got) {
    const size_t need = bytes + 1;
    if (got) *got = bytes;
    std::lock_guard<std::mutex> lk(mu_);
    if (need <= kSmallMax) {
        int c = 0;
        while ((kMinBlock << c) < need) ++c;
        const size_t block = kMinBlock << c;
        auto &fl = small_free_[c];
        if (fl.empty()) {
            const size_t slab = std::max(kSlabBytes, 16 * block);
            char *s = nullptr;
            if (slab_bytes_ + slab <= kSmallCap &&
                cudaHostAlloc((void **)&s, slab, cudaHostAllocPortable) == cudaSuccess) {
                slab_bytes_ += slab;
                ++allocs_;
                for (size_t o = slab; o >= block; o -= block) fl.push_back(s + o - block);
            } else {
                cudaGetLastError();
            }
        }
        if (!fl.empty()) {
            char *p = fl.back();
            fl.pop_back();
            live_[p] = {block, c};
            return p;
        }
    }
    const size_t mib2 = size_t(2) << 20;
    auto up = [](size_t n, size_t to) { return (n + to - 1) / to * to; };
    // best fit among the kept buffers, at most twice the size asked for
    for (const size_t fit : {need, at_least ? at_least + 1 : need}) {
        auto it = free_.lower_bound(fit);
        if (it == free_.end() || it->first > 2 * up(fit, mib2)) continue;
        char *p = it->second;
        const size_t n = it->first;
        free_.erase(it);
        free_bytes_ -= n;
        live_[p] = {n, -1};
        if (got) *got = n - 1;
        return p;
    }
    size_t step = mib2;
    while (step * 16 <= need) step *= 2;
    const size_t want = up(need, step);
    char *p = alloc_large(want);
    if (p) live_[p] = {want, -1};
    if (got) *got = want - 1;
    return p;
}

bool PinnedPool::release(char *p) {
    if (!p) return false;
    std::lock_guard<std::mutex> lk(mu_);
    auto it = live_.find(p);
    if (it == live_.end()) return false;
    const size_t n = it->second.first;
    const int c = it->second.second;
    live_.erase(it);
    if (c >= 0) {  // back to its size class; slabs are kept
        small_free_[c].push_back(p);
        return true;
    }
    free_.emplace(n, p);
    free_bytes_ += n;
    // over kKeepBytes, free the smallest kept buffers, but never the one just
    // released: a caller repeating a search whose rows alone pass the limit
    // reuses it instead of pinning gigabytes again
    while (free_bytes_ > kKeepBytes && free_.size() > 1) {
        auto victim = free_.begin();
        if (victim->second == p) ++victim;
        free_bytes_ -= victim->first;
        cudaFreeHost(victim->second);
        free_.erase(victim);
    }
    return true;
}

}  // namespace cof
