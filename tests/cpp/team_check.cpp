// CPU check of the host threads (qgate_gb300/csrc/host_team.h), built and run by
// tests/test_cpu_host_threads.py: every part runs once, for few and many parts,
// after pauses in which the helpers fall asleep, from several threads at a time,
// from within a part, and in a forked child; and a run does not wait for helpers
// that get no core (other threads spin on them all, as a BLAS's do after a call).
// Prints "ok" or what failed.
#include "host_team.h"

#include <sys/wait.h>

#include <cstdio>

using qg::HostTeam;

static bool once(int parts) {
    std::vector<std::atomic<int>> hits(parts);
    for (auto &h : hits) h = 0;
    HostTeam::run(parts, [&](int p) { hits[p].fetch_add(1); });
    for (auto &h : hits)
        if (h != 1) return false;
    return true;
}

int main() {
    for (int round = 0; round < 300; ++round)
        for (int parts : {0, 1, 2, 3, 7, 16, 61}) {
            if (!once(parts)) return printf("parts %d\n", parts), 1;
            if (round % 50 == 0) usleep(300);  // longer than the helpers look for work
        }
    std::atomic<bool> bad(false);
    std::vector<std::thread> callers;
    for (int k = 0; k < 4; ++k)
        callers.emplace_back([&] {
            for (int i = 0; i < 500; ++i)
                if (!once(5 + i % 9)) bad = true;
        });
    for (auto &t : callers) t.join();
    if (bad) return printf("several callers\n"), 1;
    std::atomic<int> inner(0);
    HostTeam::run(6, [&](int) { HostTeam::run(3, [&](int) { inner.fetch_add(1); }); });
    if (inner != 18) return printf("nested: %d\n", inner.load()), 1;
    std::atomic<bool> stop(false);
    std::vector<std::thread> spinners;
    for (int k = 0; k < 2 * (int)std::thread::hardware_concurrency(); ++k)
        spinners.emplace_back([&] {
            while (!stop.load(std::memory_order_relaxed)) {
            }
        });
    std::vector<double> us;
    for (int i = 0; i < 61; ++i) {
        usleep(300);
        const auto t = std::chrono::steady_clock::now();
        if (!once(6)) bad = true;
        us.push_back(std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t).count());
    }
    stop = true;
    for (auto &t : spinners) t.join();
    std::sort(us.begin(), us.end());
    if (bad || us[30] > 1000.) return printf("busy cores: median %.0f us\n", us[30]), 1;
    const pid_t child = fork();
    if (child == 0) _exit(once(9) ? 0 : 1);
    int status = 1;
    waitpid(child, &status, 0);
    if (status != 0) return printf("forked child\n"), 1;
    printf("ok\n");
    return 0;
}
