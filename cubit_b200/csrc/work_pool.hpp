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
            stop_ = true;
            open_.fetch_add(1);   // ends the spinning
        }
        cv_.notify_all();
        for (std::thread& t : threads_) t.join();
    }
    WorkPool(const WorkPool&) = delete;
    WorkPool& operator=(const WorkPool&) = delete;

    // Threads that can work on one job: the workers and the caller.
    unsigned width() const { return wanted_ + 1; }

    // Calls fn(piece) for every piece in [0, n), from several threads, and returns when all are done.  An exception is
    // rethrown here; with several, the one of the lowest piece.  May be called from several threads at once.
    template <typename Fn>
    void run(size_t n, Fn&& fn) {
        if (n <= 1 || !wanted_) {
            for (size_t i = 0; i < n; ++i) fn(i);
            return;
        }
        typedef typename std::remove_reference<Fn>::type Body;
        Job job;
        job.n = n;
        job.body = const_cast<void*>(static_cast<const void*>(&fn));
        job.call = [](void* body, size_t i) { (*static_cast<Body*>(body))(i); };
        {
            std::lock_guard<std::mutex> g(mu_);
            if (threads_.empty()) start();
            jobs_.push_back(&job);
            open_.fetch_add(1);
        }
        cv_.notify_one();   // a woken worker wakes the next one
        job.work(open_);
        {
            std::lock_guard<std::mutex> g(mu_);
            jobs_.erase(std::find(jobs_.begin(), jobs_.end(), &job));
        }
        // Nobody can join the job any more; those who did finish the pieces that they took.
        while (job.users.load(std::memory_order_acquire)) relax();
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
        std::atomic<size_t> next{0};
        std::atomic<unsigned> users{0};
        std::atomic<bool> drained{false};
        std::mutex error_mu;
        std::exception_ptr error;
        size_t error_at = 0;
        void work(std::atomic<int>& open) {
            for (size_t i; (i = next.fetch_add(1, std::memory_order_relaxed)) < n;) {
                try {
                    call(body, i);
                } catch (...) {
                    std::lock_guard<std::mutex> g(error_mu);
                    if (!error || i < error_at) { error = std::current_exception(); error_at = i; }
                }
            }
            if (!drained.exchange(true)) open.fetch_sub(1);   // every piece is taken: nothing for anybody to join
        }
    };

    void start() {   // mu_ is held
        for (unsigned k = 0; k < wanted_; ++k) {
            try {
                threads_.emplace_back([this] { loop(); });
            } catch (const std::system_error&) {   // no more threads to be had: go on with those that there are
                if (threads_.empty()) wanted_ = 0;
                return;
            }
        }
    }

    void loop() {
        for (;;) {
            Job* job = nullptr;
            const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(kSpinMicros);
            while (!job) {
                for (int k = 0; k < 32 && !open_.load(std::memory_order_relaxed); ++k) relax();
                const bool tired = std::chrono::steady_clock::now() > until;
                if (!tired && !open_.load(std::memory_order_relaxed)) continue;
                std::unique_lock<std::mutex> g(mu_);
                if (tired) cv_.wait(g, [this] { return stop_ || unfinished(); });
                if (stop_) return;
                if ((job = unfinished())) job->users.fetch_add(1, std::memory_order_relaxed);
            }
            cv_.notify_one();
            job->work(open_);
            job->users.fetch_sub(1, std::memory_order_release);
        }
    }
    Job* unfinished() const {
        for (Job* j : jobs_)
            if (j->next.load(std::memory_order_relaxed) < j->n) return j;
        return nullptr;
    }

    enum { kSpinMicros = 50 };
    std::atomic<unsigned> wanted_;
    std::mutex mu_;
    std::condition_variable cv_;
    std::vector<std::thread> threads_;
    std::vector<Job*> jobs_;
    std::atomic<int> open_{0};   // jobs with pieces left to take: what idle workers look at without the lock
    bool stop_ = false;
};

}  // namespace cubit
