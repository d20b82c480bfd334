// pinned_pool.hpp -- the free list of a context's page-locked result blocks. Host code only; the
// allocation itself is the caller's (Alloc, Free), so a check of the list needs no device.
#pragma once
#include <cstddef>
#include <map>
#include <mutex>

namespace zk {

// Allocating and freeing page-locked memory can wait for the whole device, so blocks come in a few
// sizes, powers of two from kSmallest on (the targets of every single MSM fit the smallest), and
// are kept for reuse. The list holds at most kKeep bytes: a block given back beyond that is freed.
// Thread-safe.
class PinnedPool {
   public:
    static constexpr size_t kSmallest = (size_t)64 << 10;
    static constexpr size_t kKeep = (size_t)256 << 20;

    static size_t size_class(size_t bytes) {
        size_t s = kSmallest;
        while (s < bytes) s *= 2;
        return s;
    }

    // A block of size_class(bytes), from the list or of alloc(size); null when alloc says so.
    template <class Alloc>
    void* take(size_t bytes, Alloc&& alloc) {
        const size_t size = size_class(bytes);
        {
            std::lock_guard<std::mutex> g(mu_);
            auto it = free_.find(size);
            if (it != free_.end()) {
                void* p = it->second;
                free_.erase(it);
                kept_ -= size;
                return p;
            }
        }
        return alloc(size);
    }

    // `bytes` as taken.
    template <class Free>
    void give(void* p, size_t bytes, Free&& release) {
        if (p == nullptr) return;
        const size_t size = size_class(bytes);
        {
            std::lock_guard<std::mutex> g(mu_);
            if (kept_ + size <= kKeep) {
                free_.emplace(size, p);
                kept_ += size;
                return;
            }
        }
        release(p);
    }

    template <class Free>
    void clear(Free&& release) {
        std::lock_guard<std::mutex> g(mu_);
        for (auto& kv : free_) release(kv.second);
        free_.clear();
        kept_ = 0;
    }

   private:
    std::mutex mu_;
    std::multimap<size_t, void*> free_;  // size -> block
    size_t kept_ = 0;
};

}  // namespace zk
