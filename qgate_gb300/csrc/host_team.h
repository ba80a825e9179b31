// Host threads for short pieces of work (copies out of staging buffers, block
// operands).  Only as many are woken as have work: an OpenMP region of fewer
// threads than the last one makes the runtime end the others, and the next region
// that wants them all pays 150 to 230 us for new ones (Grace), while waking the
// whole team for a 1 MB copy takes longer (30 us) than copying it alone (21 us).
#pragma once

#include <omp.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace qg {

class HostTeam {
public:
    // Calls f(0), .., f(parts - 1), each once, on up to omp_get_max_threads()
    // threads, the caller's among them; f must not throw.  Called while the helpers
    // are at work (by another thread, or from within f) or from an OpenMP region, it
    // makes all the calls itself.
    template <class F> static void run(int parts, const F &f) {
        std::atomic<bool> &taken = in_run();
        if (parts > 1 && !omp_in_parallel() && !taken.exchange(true)) {
            HostTeam &t = team();
            const int helpers = t.ready(std::min(parts, omp_get_max_threads()) - 1);
            std::atomic<int> next(0), busy(helpers);
            const Job job = {[](const void *fn, int part) { (*(const F *)fn)(part); }, &f, parts,
                             &next, &busy};
            for (int k = 0; k < helpers; ++k) t.workers_[k]->start(&job);
            job.work();
            while (busy.load(std::memory_order_acquire) != 0) std::this_thread::yield();
            taken.store(false);
            return;
        }
        for (int p = 0; p < parts; ++p) f(p);
    }

private:
    struct Job {
        void (*call)(const void *, int);
        const void *fn;
        int parts;
        std::atomic<int> *next, *busy;
        void work() const {
            for (int p; (p = next->fetch_add(1, std::memory_order_relaxed)) < parts;) call(fn, p);
        }
    };
    // Looks for its next job for 100 us (pieces often follow one another), then sleeps.
    struct Worker {
        std::mutex m;
        std::condition_variable cv;
        std::atomic<const Job *> job{nullptr};
        std::atomic<bool> asleep{false};
        void start(const Job *j) {
            job.store(j);
            if (!asleep.load()) return;  // (it looks for the job after saying that it sleeps)
            std::lock_guard<std::mutex> lk(m);
            cv.notify_one();
        }
        void loop() {
            for (;;) {
                const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(100);
                while (!job.load() && std::chrono::steady_clock::now() < until)
                    std::this_thread::yield();
                if (!job.load()) {
                    std::unique_lock<std::mutex> lk(m);
                    asleep.store(true);
                    cv.wait(lk, [&] { return job.load() != nullptr; });
                    asleep.store(false);
                }
                const Job *j = job.exchange(nullptr);
                j->work();
                j->busy->fetch_sub(1, std::memory_order_release);  // the job ends with it
            }
        }
    };

    static std::atomic<bool> &in_run() {
        static std::atomic<bool> taken{false};
        return taken;
    }
    // The process's team: its threads wait for ever and end with the process.  A
    // forked child starts its own.
    static HostTeam &team() {
        static HostTeam *t = nullptr;
        static pid_t owner = 0;
        if (!t || owner != getpid()) {
            t = new HostTeam();
            owner = getpid();
        }
        return *t;
    }
    // How many of n helpers there are, started as far as the system allows.
    int ready(int n) {
        while ((int)workers_.size() < n) {
            Worker *w = new Worker();
            try {
                std::thread([w] { w->loop(); }).detach();
            } catch (const std::system_error &) {
                delete w;
                break;
            }
            workers_.push_back(w);
        }
        return std::min(n, (int)workers_.size());
    }
    std::vector<Worker *> workers_;
};

}  // namespace qg
