// A context's device memory: what its budget admits, and freed blocks kept for
// the next allocations.  The device allocator is behind two functions, so the
// rules can be tested without a GPU.
//
// Kept blocks: a 4.3 GB octree's cudaMalloc and cudaFree take 0.6 and 1.8 ms,
// more than half of its build's kernels.  At most `cap` bytes are kept, the
// oldest given back first; all of them when an allocation fails or the context
// goes.  A block is kept only when nothing on the device uses it any more.
//
// With a budget, `used` plus what is kept never exceeds it, during an
// allocation neither: blocks are allocated at the size that was asked for,
// only a block of exactly that size is taken again, and room is made before
// the device allocator is called.  Without one, sizes are rounded up to a 16th
// of their power of two and a block up to an eighth larger serves, so that the
// next octree of about the same size finds the last one's blocks.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace xn {

class BlockPool {
public:
    struct Api {
        int (*alloc)(void** p, uint64_t bytes);  // 0 or an error > 0
        void (*release)(void* p);
        int out_of_memory;  // alloc's error when memory is short
    };
    static constexpr int OVER_BUDGET = -1;
    static constexpr uint64_t SMALLEST = 64 << 10;  // smaller blocks are not kept

    uint64_t budget = 0;  // 0: none; set before the first allocation, like cap
    uint64_t cap = 0;
    std::atomic<uint64_t> used{0};  // bytes asked for and not yet freed

    explicit BlockPool(const Api& a) : api(a) {}

    // An allocation that does not go through the pool, tried again without the
    // kept blocks: f returns 0 or the allocator's error.
    template <class F>
    auto with_room(F f) {
        auto e = f();
        if ((int)e == api.out_of_memory) {
            trim(0);
            e = f();
        }
        return e;
    }

    // 0, OVER_BUDGET or the allocator's error.
    int alloc(void** p, uint64_t bytes) {
        *p = nullptr;
        const uint64_t size = budget ? bytes : rounded(bytes);
        {
            std::lock_guard<std::mutex> lk(mu);
            if (!admit(bytes)) return OVER_BUDGET;
            const uint64_t most = budget ? size : size + size / 8;
            size_t best = kept.size();
            for (size_t i = 0; i < kept.size(); ++i)
                if (kept[i].bytes >= size && kept[i].bytes <= most &&
                    (best == kept.size() || kept[i].bytes < kept[best].bytes))
                    best = i;
            if (best < kept.size()) {
                *p = kept[best].p;
                kept_bytes -= kept[best].bytes;
                sizes[*p] = kept[best].bytes;
                kept.erase(kept.begin() + (std::ptrdiff_t)best);
                return 0;
            }
            make_room();
        }
        uint64_t got = 0;
        const int e = with_room([&] {  // the second time without the rounding
            got = got ? bytes : size;
            return api.alloc(p, got);
        });
        std::lock_guard<std::mutex> lk(mu);
        if (e) {
            *p = nullptr;
            used -= bytes;
            return e;
        }
        sizes[*p] = got;
        return 0;
    }

    // idle: nothing on the device uses the block any more.
    void free(void* p, uint64_t bytes, bool idle) {
        {
            std::lock_guard<std::mutex> lk(mu);
            auto it = sizes.find(p);
            const uint64_t size = it == sizes.end() ? 0 : it->second;
            if (it != sizes.end()) sizes.erase(it);
            const uint64_t rest = used.load() - bytes;
            const uint64_t room = budget ? std::min(cap, budget - rest) : cap;
            if (idle && size >= SMALLEST && size <= room) {
                trim_locked(room - size);
                kept.push_back({p, size});
                kept_bytes += size;
                used -= bytes;
                return;
            }
        }
        api.release(p);
        used -= bytes;
    }

    // Memory that the caller allocates itself (arrays) is counted and makes
    // room the same way: false where the budget does not admit it.
    bool reserve(uint64_t bytes) {
        std::lock_guard<std::mutex> lk(mu);
        if (!admit(bytes)) return false;
        make_room();
        return true;
    }
    void unreserve(uint64_t bytes) { used -= bytes; }

    // Gives blocks back until at most `keep` bytes are kept.
    void trim(uint64_t keep) {
        std::lock_guard<std::mutex> lk(mu);
        trim_locked(keep);
    }

private:
    struct Block {
        void* p;
        uint64_t bytes;
    };
    const Api api;
    std::mutex mu;
    std::vector<Block> kept;                    // oldest first
    std::unordered_map<void*, uint64_t> sizes;  // of the blocks in use
    uint64_t kept_bytes = 0;

    static uint64_t rounded(uint64_t bytes) {
        uint64_t unit = 512;
        while (unit * 32 <= bytes) unit <<= 1;
        return (bytes + unit - 1) / unit * unit;
    }
    bool admit(uint64_t bytes) {
        if (budget && bytes > budget - used.load()) return false;
        used += bytes;
        return true;
    }
    void make_room() {
        if (budget) trim_locked(budget - used.load());
    }
    void trim_locked(uint64_t keep) {
        size_t n = 0;
        while (kept_bytes > keep && n < kept.size()) {
            api.release(kept[n].p);
            kept_bytes -= kept[n++].bytes;
        }
        kept.erase(kept.begin(), kept.begin() + (std::ptrdiff_t)n);
    }
};

}  // namespace xn
