// CPU check of the tensor-stage planner on gates with up to ten lanes (built and
// run by tests/test_cpu_wide_gates.py): every gate is planned once, no stage
// holds a gate with more lanes in its tile than a fused block has, and the
// blocks of every stage are finite.  Prints "<check> <value>" lines.
#include "tcplan.cpp"

#include <cstdio>
#include <random>

using namespace qg;

int main() {
    std::mt19937 rng(5);
    int wide = 0, stages = 0, bad = 0;
    for (int trial = 0; trial < 40; ++trial) {
        const int n = 13 + trial % 5;
        const bool cross = trial & 1;
        std::vector<PendingGate> gates(60);
        for (auto &g : gates) {
            std::vector<int> lanes(n);
            for (int i = 0; i < n; ++i) lanes[i] = i;
            std::shuffle(lanes.begin(), lanes.end(), rng);
            g.target = lanes[0];
            g.controls.assign(lanes.begin() + 1, lanes.begin() + 1 + rng() % 10);
            const bool diag = rng() % 2;
            const double v[8] = {diag ? 1. : 0., 0, diag ? 0. : 1., 0,
                                 diag ? 0. : 1., 0, diag ? -1. : 0., 0};
            memcpy(g.m.v, v, sizeof(v));
            g.diag = is_diag(g.m);
        }
        std::vector<const PendingGate *> rem;
        for (auto &g : gates) rem.push_back(&g);
        size_t done = 0;
        while (!rem.empty()) {
            const unsigned long long q0 = gate_qmask(*rem[0]);
            if (__builtin_popcountll(q0 | 15ull) > 12 || __builtin_popcountll(q0) > kTcBlockLanes) {
                ++wide;
                ++done;
                rem.erase(rem.begin());
                continue;
            }
            unsigned long long S = plan_stage_lanes(rem, 15ull, 12, cross, kMaxTensorStageGates);
            std::vector<const PendingGate *> take, keep;
            stage_take(rem, S, rem.size(), &take, &keep, cross, kMaxTensorStageGates);
            if (take.empty()) {
                ++bad;
                break;
            }
            for (int q = 0; q < n && __builtin_popcountll(S) < 12; ++q) S |= 1ULL << q;
            for (auto *g : take)
                if (__builtin_popcountll(gate_qmask(*g) & S) > kTcBlockLanes) ++bad;
            size_t held = 0;
            if (!bad)
                for (auto &b : tc_blocks(take, tile_lanes_of(S, n))) held += b.second.size();
            if (held != take.size()) ++bad;
            done += take.size();
            ++stages;
            rem.swap(keep);
        }
        if (done != gates.size()) ++bad;
    }
    printf("wide %d\nstages %d\nbad %d\n", wide, stages, bad);
    return 0;
}
