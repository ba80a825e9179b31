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
            Job *job = new Job{[](const void *fn, int part) { (*(const F *)fn)(part); }, &f, parts};
            for (int k = 0; k < helpers; ++k) {
                job->refs.fetch_add(1, std::memory_order_relaxed);
                t.workers_[k]->start(job);
            }
            job->work();
            // helpers that have not come to it (the cores are busy) are not waited for
            for (int k = 0; k < helpers; ++k)
                if (Job *left = t.workers_[k]->job.exchange(nullptr)) left->drop();
            while (job->done.load(std::memory_order_acquire) < parts) std::this_thread::yield();
            job->drop();
            taken.store(false);
            return;
        }
        for (int p = 0; p < parts; ++p) f(p);
    }

private:
    // A job lives until its last helper has seen it; f is called only while run waits
    // for the part.
    struct Job {
        void (*call)(const void *, int);
        const void *fn;
        int parts;
        std::atomic<int> next{0}, done{0}, refs{1};
        void work() {
            for (int p; (p = next.fetch_add(1, std::memory_order_relaxed)) < parts;) {
                call(fn, p);
                done.fetch_add(1, std::memory_order_release);
            }
        }
        void drop() {
            if (refs.fetch_sub(1, std::memory_order_acq_rel) == 1) delete this;
        }
    };
    // Looks for its next job for 100 us (pieces often follow one another), then sleeps.
    struct Worker {
        std::mutex m;
        std::condition_variable cv;
        std::atomic<Job *> job{nullptr};
        std::atomic<bool> asleep{false};
        void start(Job *j) {
            job.store(j);
            // Not under m: a worker on its way to sleep may miss this one, and run then
            // takes the job back.
            if (asleep.load()) cv.notify_one();
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
                if (Job *j = job.exchange(nullptr)) {  // (not taken back meanwhile)
                    j->work();
                    j->drop();
                }
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
