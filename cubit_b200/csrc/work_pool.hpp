// Host worker threads that a context keeps for the parts of a call that run on the CPU: text, and copies between
// the caller's buffers and the pinned staging area.
//
// A job is a number of independent pieces; the calling thread works on them too, so a job ends even when every worker is
// busy elsewhere (or does not exist: a host with one core, a forked child).  Starting a thread costs about 12 us and a
// sleeping one several times that to wake on a virtual machine, so the threads outlive the calls, and one that runs out
// of work keeps looking for a while before it goes to sleep: the copies of one host batch follow each other within that time.
#pragma once
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <type_traits>
#include <vector>

namespace cubit {

class WorkPool {
public:
    explicit WorkPool(unsigned workers) : wanted_(workers) {}
    ~WorkPool() {
        {
            std::lock_guard<std::mutex> g(mu_);
            stop_.store(true);
        }
        cv_.notify_all();
        for (std::thread& t : threads_) t.join();
    }
    WorkPool(const WorkPool&) = delete;
    WorkPool& operator=(const WorkPool&) = delete;

    // Threads that can work on one job: the workers and the caller.
    unsigned width() const { return wanted_ + 1; }

    // While one of these lives, workers without work keep looking for longer: a call that waits for the GPU between its
    // jobs finds them awake (asleep, they cost a batch of 9 Mi words 3 of 8 ms).
    class Awake {
    public:
        explicit Awake(WorkPool& pool) : pool_(pool) { pool_.awake_.fetch_add(1, std::memory_order_relaxed); }
        ~Awake() { pool_.awake_.fetch_sub(1, std::memory_order_relaxed); }
        Awake(const Awake&) = delete;
        Awake& operator=(const Awake&) = delete;
    private:
        WorkPool& pool_;
    };

    // Calls fn(piece) for every piece in [0, n), from several threads, and returns when all are done.  An exception is
    // rethrown here; with several, the one of the lowest piece.  May be called from several threads at once.
    template <typename Fn>
    void run(size_t n, Fn&& fn) {
        typedef typename std::remove_reference<Fn>::type Body;
        Job job;
        job.n = n;
        job.body = const_cast<void*>(static_cast<const void*>(&fn));
        job.call = [](void* body, size_t i) { (*static_cast<Body*>(body))(i); };
        Slot* slot = n > 1 && wanted_ && started() ? publish(&job) : nullptr;
        job.work(open_, slot != nullptr);
        if (slot) {
            // Nobody can join the job any more once it is withdrawn; those who did finish the pieces that they took.
            slot->job.store(nullptr);
            while (slot->users.load()) relax();
            slot->taken.store(false, std::memory_order_release);
        }
        if (job.error) std::rethrow_exception(job.error);
    }

    // The number of pieces of at least `grain` items that n items are worth cutting into.
    size_t pieces(size_t n, size_t grain, size_t per_thread = 1) const {
        return std::max<size_t>(1, std::min<size_t>(n / std::max<size_t>(grain, 1), (size_t)width() * per_thread));
    }

    // The processor's hint for a waiting loop.
    static void relax() {
#if defined(__x86_64__) || defined(__i386__)
        __builtin_ia32_pause();
#else
        std::this_thread::yield();
#endif
    }

private:
    struct Job {
        size_t n = 0;
        void* body = nullptr;
        void (*call)(void*, size_t) = nullptr;
        alignas(64) std::atomic<size_t> next{0};
        std::atomic<bool> drained{false};
        std::mutex error_mu;
        std::exception_ptr error;
        size_t error_at = 0;
        void work(std::atomic<int>& open, bool published) {
            for (size_t i; (i = next.fetch_add(1, std::memory_order_relaxed)) < n;) {
                try {
                    call(body, i);
                } catch (...) {
                    std::lock_guard<std::mutex> g(error_mu);
                    if (!error || i < error_at) { error = std::current_exception(); error_at = i; }
                }
            }
            if (published && !drained.exchange(true)) open.fetch_sub(1);   // every piece is taken: nothing for anybody to join
        }
    };
    // Where a job is found.  A worker counts itself in before it looks whether the job is still there, the caller waits
    // for the count after it has taken the job away: the job outlives everybody who works on it.
    struct alignas(64) Slot {
        std::atomic<bool> taken{false};
        std::atomic<Job*> job{nullptr};
        std::atomic<unsigned> users{0};
    };

    bool started() {
        if (started_.load(std::memory_order_acquire)) return true;
        std::lock_guard<std::mutex> g(mu_);
        for (unsigned k = (unsigned)threads_.size(); k < wanted_; ++k) {
            try {
                threads_.emplace_back([this] { loop(); });
            } catch (const std::system_error&) {   // no more threads to be had: go on with those that there are
                wanted_ = k;
            }
        }
        started_.store(true, std::memory_order_release);
        return wanted_ > 0;
    }

    Slot* publish(Job* job) {   // null when too many jobs are open already: the caller does this one alone
        for (Slot& s : slots_) {
            if (s.taken.load(std::memory_order_relaxed) || s.taken.exchange(true)) continue;
            open_.fetch_add(1);
            s.job.store(job);
            wake();
            return &s;
        }
        return nullptr;
    }
    void wake() {   // one sleeper; it wakes the next
        if (!sleeping_.load()) return;
        std::lock_guard<std::mutex> g(mu_);
        cv_.notify_one();
    }

    void loop() {
        while (!stop_.load(std::memory_order_relaxed)) {
            if (join_one()) continue;
            const auto from = std::chrono::steady_clock::now();
            while (!open_.load(std::memory_order_relaxed) && !stop_.load(std::memory_order_relaxed)) {
                for (int k = 0; k < 32 && !open_.load(std::memory_order_relaxed); ++k) relax();
                const auto most = std::chrono::microseconds(awake_.load(std::memory_order_relaxed) ? kAwakeMicros : kSpinMicros);
                if (std::chrono::steady_clock::now() - from < most) continue;
                std::unique_lock<std::mutex> g(mu_);
                sleeping_.fetch_add(1);
                cv_.wait(g, [this] { return stop_.load() || open_.load() > 0; });
                sleeping_.fetch_sub(1);
                break;
            }
        }
    }
    bool join_one() {
        for (Slot& s : slots_) {
            if (!s.job.load(std::memory_order_relaxed)) continue;
            s.users.fetch_add(1);
            Job* const job = s.job.load();
            const bool worth = job && job->next.load(std::memory_order_relaxed) < job->n;
            if (worth) {
                wake();
                job->work(open_, true);
            }
            s.users.fetch_sub(1);
            if (worth) return true;
        }
        return false;
    }

    enum { kSpinMicros = 50, kAwakeMicros = 1000, kSlots = 8 };
    std::atomic<unsigned> wanted_;
    std::mutex mu_;
    std::condition_variable cv_;
    std::vector<std::thread> threads_;
    Slot slots_[kSlots];
    std::atomic<int> open_{0};        // jobs with pieces left to take: what idle workers look at
    std::atomic<int> sleeping_{0};
    std::atomic<int> awake_{0};
    std::atomic<bool> started_{false}, stop_{false};
};

}  // namespace cubit
