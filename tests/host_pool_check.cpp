// Host check of pyzkp_gb300/csrc/host_pool.hpp: workers woken ahead of a run hold nobody else out
// of the pool, go back to sleep when the run comes late, and mixed runs of several threads execute
// every task once. Exit 0 when all hold. Built and run by tests/test_host_pool.py under a time limit.
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <vector>

#include "../pyzkp_gb300/csrc/host_pool.hpp"

using Clock = std::chrono::steady_clock;
using us = std::chrono::microseconds;
static std::atomic<int> bad{0};

static void check(const char* what, bool ok) {
    if (!ok && bad.fetch_add(1) < 10) std::printf("%s\n", what);
}

struct Tasks {
    std::unique_ptr<std::atomic<int>[]> ran;
    size_t n;
    explicit Tasks(size_t count) : ran(new std::atomic<int>[count]()), n(count) {}
    std::function<void(size_t)> fn() {
        return [this](size_t i) { ran[i].fetch_add(1); };
    }
    bool once() const {
        for (size_t i = 0; i < n; i++)
            if (ran[i].load() != 1) return false;
        return true;
    }
};

// Waits up to a second for the number of awake workers.
template <class Cond>
static bool settles(Cond&& cond) {
    const auto end = Clock::now() + std::chrono::seconds(1);
    while (!cond())
        if (Clock::now() >= end) return false;
        else std::this_thread::yield();
    return true;
}

int main() {
    zk::HostPool& pool = zk::HostPool::get();
    const size_t workers = std::min<size_t>(std::max(1u, std::thread::hardware_concurrency()), 16) - 1;
    {  // workers wake, wait, run, and sleep when the announcement ends
        Tasks t(9);
        {
            zk::HostPool::Expect e(pool, 4, us(5000000));
            check("no worker woke", workers == 0 || settles([&] { return pool.awake() > 0; }));
            pool.run_with(9, t.fn(), [] {}, 4);
            check("tasks of an announced run", t.once());
        }
        check("workers stay awake", settles([&] { return pool.awake() == 0; }));
    }
    {  // a run that comes late, or never, does not keep them awake
        zk::HostPool::Expect e(pool, 4, us(2000));
        std::this_thread::sleep_for(us(4000));
        check("workers stay awake past the limit", settles([&] { return pool.awake() == 0; }));
        Tasks t(9);
        pool.run_with(9, t.fn(), [] {}, 4);
        check("tasks of a late run", t.once());
    }
    // a call that waits for its data while another caller's run is what brings it: neither waits for the other
    for (size_t count : {2, 16, 40}) {
        Tasks mine(8), other(count);
        std::atomic<bool> waiting{false};
        std::thread b([&] {
            while (!waiting.load()) std::this_thread::yield();
            pool.run(count, other.fn());
        });
        zk::HostPool::Expect e(pool, 4, us(1000000));
        waiting.store(true);
        while (!other.once()) std::this_thread::yield();
        pool.run_with(8, mine.fn(), [] {}, 4);
        b.join();
        check("tasks beside another run", mine.once());
    }
    {  // a busy pool is not waited for, and one Expect at a time wakes workers
        Tasks outer(4), inner(3);
        bool refused = false, owned = false;
        pool.run_with(4, outer.fn(), [&] {
            std::thread([&] { refused = !pool.run_with(3, inner.fn(), [&] { owned = true; }, 4, true); }).join();
        });
        check("a busy pool was not refused", refused && !owned && inner.ran[0] + inner.ran[1] + inner.ran[2] == 0);
        check("tasks of the outer run", outer.once());
        check("a free pool was refused", pool.run_with(3, inner.fn(), [&] { owned = true; }, 4, true) && owned && inner.once());
        zk::HostPool::Expect a(pool, 1, us(5000000));
        check("no worker woke", workers == 0 || settles([&] { return pool.awake() > 0; }));
        zk::HostPool::Expect b(pool, 4, us(5000000));
        std::this_thread::sleep_for(us(2000));
        check("a second Expect woke workers", pool.awake() <= 2);
    }
    check("workers stay awake", settles([&] { return pool.awake() == 0; }));
    // mixed runs from several threads
    std::vector<std::thread> ts;
    for (int k = 0; k < 6; k++)
        ts.emplace_back([&, k] {
            for (int i = 0; i < 400; i++) {
                Tasks t(1 + (i * 7 + k) % 60);
                if (k % 2) {
                    zk::HostPool::Expect e(pool, 4, us(i % 3 * 50));
                    std::this_thread::sleep_for(us(i % 5 * 20));
                    if (i % 2 || !pool.run_with(t.n, t.fn(), [] {}, 4, true)) pool.run_with(t.n, t.fn(), [] {}, 4);
                } else {
                    pool.run(t.n, t.fn());
                }
                check("a task did not run once", t.once());
            }
        });
    for (auto& t : ts) t.join();
    check("workers stay awake", settles([&] { return pool.awake() == 0; }));
    std::printf("%d failed\n", bad.load());
    return bad.load() != 0;
}
