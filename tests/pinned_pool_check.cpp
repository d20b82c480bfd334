// Host check of pyzkp_gb300/csrc/pinned_pool.hpp with a counting allocator: sizes of one class share
// a block, the list stays within its limit, and threads never hold one block twice. Exit 0 when all
// hold. Built and run by tests/test_pinned_pool.py.
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "../pyzkp_gb300/csrc/pinned_pool.hpp"

static std::atomic<long> allocs{0}, frees{0};
static int bad = 0;

static void* alloc(size_t) {
    allocs++;
    return std::malloc(64);
}
static void release(void* p) {
    frees++;
    std::free(p);
}
static void check(const char* what, bool ok) {
    if (!ok && bad++ < 10) std::printf("%s\n", what);
}

int main() {
    using zk::PinnedPool;
    {
        PinnedPool pool;
        // the targets of single MSMs: up to 33 sets of 18 G2 points and the entry count
        for (size_t bytes = 1; bytes <= 64 << 10; bytes += 997) {
            void* p = pool.take(bytes, alloc);
            pool.give(p, bytes, release);
        }
        check("a new size of the smallest class allocated", allocs == 1);
        for (size_t bytes : {(size_t)65537, (size_t)100000, (size_t)131072}) pool.give(pool.take(bytes, alloc), bytes, release);
        check("sizes of one class did not share", allocs == 2);
        check("classes", PinnedPool::size_class(1) == PinnedPool::kSmallest && PinnedPool::size_class(65536) == 65536 &&
                             PinnedPool::size_class(65537) == 131072);
        void* none = pool.take((size_t)1 << 30, [](size_t) -> void* { return nullptr; });
        check("a failed allocation", none == nullptr);
        pool.give(none, (size_t)1 << 30, release);
        pool.clear(release);
        check("clear", frees == allocs);
    }
    {
        PinnedPool pool;
        allocs = frees = 0;
        std::vector<void*> held;
        const size_t bytes = (size_t)8 << 20, fit = PinnedPool::kKeep / bytes;
        for (size_t i = 0; i < 3 * fit; i++) held.push_back(pool.take(bytes, alloc));
        for (void* p : held) pool.give(p, bytes, release);
        check("the list is not bounded", frees == (long)(2 * fit));
        for (size_t i = 0; i < fit; i++) held[i] = pool.take(bytes, alloc);
        check("kept blocks were not reused", allocs == (long)(3 * fit));
        for (size_t i = 0; i < fit; i++) pool.give(held[i], bytes, release);
        pool.clear(release);
        check("clear", frees == allocs);
    }
    {
        PinnedPool pool;
        std::atomic<int> twice{0};
        std::vector<std::thread> ts;
        for (int k = 0; k < 4; k++)
            ts.emplace_back([&, k] {
                for (int i = 0; i < 20000; i++) {
                    const size_t bytes = (size_t)1 << (10 + (i + k) % 9);
                    auto* p = static_cast<volatile int*>(pool.take(bytes, [](size_t) -> void* { return std::calloc(16, 4); }));
                    p[0] = p[0] + 1;
                    if (p[0] != 1) twice++;
                    p[0] = 0;
                    pool.give((void*)p, bytes, [](void* q) { std::free(q); });
                }
            });
        for (auto& t : ts) t.join();
        check("a block was held twice", twice == 0);
        pool.clear([](void* q) { std::free(q); });
    }
    std::printf("%d failed\n", bad);
    return bad != 0;
}
