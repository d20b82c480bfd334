// host_pool.hpp -- the library's pool of host threads (MSM window sums). Host code only.
#pragma once
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <mutex>
#include <thread>

namespace zk {

// A persistent pool of host threads for the combination step (created on first use,
// never destroyed: its threads sleep between jobs). run() executes fn(0 .. count-1) on the
// calling thread and on at most count - 1 woken workers, and returns when every task is
// done -- not when every worker has woken: a late worker finds no task left and sleeps
// again. Tasks are claimed from one atomic ticket (generation | count | next index), so a
// worker can only claim a task of the run in progress; calls are serialised.
class HostPool {
    using Clock = std::chrono::steady_clock;

   public:
    static HostPool& get() {
        static HostPool* pool = new HostPool();
        return *pool;
    }

    void run(size_t count, const std::function<void(size_t)>& fn) {
        if (count == 1 || workers_ == 0) {  // no helper: no shared state, no lock
            for (size_t i = 0; i < count; i++) fn(i);
            return;
        }
        run_with(count, fn, [] {});
    }

    // run() in which the calling thread first executes own(): own() may take tasks itself
    // through run_one() (the same ticket, so in the same index order as the workers), e.g.
    // to consume results in order and compute whichever no worker has taken yet. Returns true;
    // if_free: returns false with nothing done when another run is in progress (for a few tasks:
    // by the time that one is over, the calling thread would be through with them).
    template <class Own>
    bool run_with(size_t count, const std::function<void(size_t)>& fn, Own&& own, size_t max_helpers = ~size_t(0),
                  bool if_free = false) {
        if (count == 0 || count > kMaxTasks) {
            for (size_t i = 0; i < count; i++) fn(i);
            own();
            return true;
        }
        std::unique_lock<std::mutex> serial(run_mu_, std::try_to_lock);
        if (!serial.owns_lock()) {
            if (if_free) return false;
            serial.lock();
        }
        gen_ = (gen_ + 1) & 0xffffu;
        fn_ = &fn;
        done_.store(0, std::memory_order_relaxed);
        ticket_.store(gen_ << 48 | (uint64_t)count << 24, std::memory_order_release);
        size_t helpers = std::min(std::min(count - 1, workers_), max_helpers);
        // those awake see the ticket without a wake-up, which the caller would pay for before own(): with
        // half of the helpers awake there is none
        const size_t up = awake();
        helpers = 2 * up >= helpers ? 0 : helpers - up;
        if (helpers > 0) {
            // the caller wakes up to kFanout workers and each woken worker up to kFanout more
            // (a wake-up is a system call of a few microseconds: a tree of them instead of a
            // row on the caller)
            const size_t first = std::min(helpers, kFanout);
            pending_.store((int64_t)(helpers - first), std::memory_order_relaxed);
            {
                std::lock_guard<std::mutex> g(mu_);
                wake_++;
            }
            for (size_t i = 0; i < first; i++) cv_.notify_one();
        }
        own();
        work();
        // the tasks still running were claimed by awake workers; the wait re-checks every
        // millisecond, so even a lost wakeup of the condition variable only costs that much
        std::unique_lock<std::mutex> g(mu_);
        while (done_.load(std::memory_order_acquire) < count)
            done_cv_.wait_for(g, std::chrono::milliseconds(1),
                              [&] { return done_.load(std::memory_order_acquire) >= count; });
        return true;
    }

    // Wakes up to `helpers` workers ahead of a run that this thread is about to start: they wait awake
    // for tasks (of any caller's run) while the Expect lives, at most for `limit`. Holds nothing:
    // other runs go on as without it.
    class Expect {
       public:
        Expect(HostPool& pool, size_t helpers, std::chrono::microseconds limit) : pool_(pool) {
            // one at a time: with several callers about, the workers that one of them woke serve all
            size_t none = 0;
            if (helpers == 0 || !pool_.expected_.compare_exchange_strong(none, helpers, std::memory_order_acq_rel)) return;
            mine_ = true;
            pool_.until_.store((Clock::now() + limit).time_since_epoch().count(), std::memory_order_release);
            helpers = std::min(helpers, pool_.workers_);
            const size_t first = std::min(helpers, kFanout);
            const int64_t rest = (int64_t)(helpers - first);  // passed on, beside what a run has left to pass on
            int64_t p = pool_.pending_.load(std::memory_order_relaxed);
            while (p < rest && !pool_.pending_.compare_exchange_weak(p, rest, std::memory_order_acq_rel)) {
            }
            {
                std::lock_guard<std::mutex> g(pool_.mu_);
                pool_.wake_++;
            }
            for (size_t i = 0; i < first; i++) pool_.cv_.notify_one();
        }
        ~Expect() {
            if (mine_) pool_.expected_.store(0, std::memory_order_release);
        }
        Expect(const Expect&) = delete;
        Expect& operator=(const Expect&) = delete;

       private:
        HostPool& pool_;
        bool mine_ = false;
    };

    // Workers that wait awake.
    size_t awake() const { return awake_.load(std::memory_order_acquire); }

    // Claim and run the next task of the run in progress; false if none is left.
    bool run_one() {
        for (;;) {
            uint64_t cur = ticket_.load(std::memory_order_acquire);
            const uint64_t count = (cur >> 24) & kMaxTasks, i = cur & kMaxTasks;
            if (i >= count) return false;
            if (!ticket_.compare_exchange_weak(cur, cur + 1, std::memory_order_acq_rel)) continue;
            (*fn_)(i);
            if (done_.fetch_add(1, std::memory_order_acq_rel) + 1 == count) {
                std::lock_guard<std::mutex> g(mu_);
                done_cv_.notify_all();
            }
            return true;
        }
    }

    // Whether task i of the run in progress has been claimed.
    bool claimed(size_t i) const { return (ticket_.load(std::memory_order_acquire) & kMaxTasks) > i; }

   private:
    static constexpr size_t kMaxTasks = (1u << 24) - 1;

    HostPool() {
        const size_t hw = std::max<size_t>(1, std::thread::hardware_concurrency());
        workers_ = std::min<size_t>(hw, 16) - 1;
        for (size_t i = 0; i < workers_; i++) std::thread([this] { loop(); }).detach();
    }

    void loop() {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> g(mu_);
                cv_.wait(g, [&] { return wake_ != seen; });
                seen = wake_;
            }
            for (size_t i = 0; i < kFanout; i++)
                if (pending_.fetch_sub(1, std::memory_order_acq_rel) > 0) cv_.notify_one();
            work();
            // the run that an Expect announces: its wake-up takes 10 - 20 us, as long as two or three window sums
            // (twice as many may stay: some of those asked for may still be on their way to sleep)
            if (awake_.fetch_add(1, std::memory_order_acq_rel) < 2 * expected_.load(std::memory_order_acquire))
                while (expected_.load(std::memory_order_acquire) != 0 &&
                       Clock::now().time_since_epoch().count() < until_.load(std::memory_order_acquire))
                    if (!run_one()) std::this_thread::yield();
            awake_.fetch_sub(1, std::memory_order_acq_rel);
        }
    }

    // Claim and run tasks while the ticket has some left. A successful claim of task i means
    // the run that published the ticket is still waiting for task i, so fn_ is its function.
    void work() {
        while (run_one()) {
        }
    }

    size_t workers_ = 0;
    std::mutex run_mu_, mu_;
    std::condition_variable cv_, done_cv_;
    uint64_t wake_ = 0;  // under mu_
    uint64_t gen_ = 0;   // under run_mu_
    static constexpr size_t kFanout = 2;
    // on cache lines of their own: workers that wait awake read the ticket and the announcement
    // all the time
    alignas(128) const std::function<void(size_t)>* fn_ = nullptr;
    std::atomic<int64_t> pending_{0};  // wake-ups the woken workers still have to pass on
    alignas(128) std::atomic<uint64_t> ticket_{0};
    alignas(128) std::atomic<size_t> done_{0};
    alignas(128) std::atomic<size_t> expected_{0};  // workers that the Expect alive asked for
    std::atomic<Clock::rep> until_{0};              // when they go to sleep all the same
    alignas(128) std::atomic<size_t> awake_{0};     // workers that wait awake
};

}  // namespace zk
