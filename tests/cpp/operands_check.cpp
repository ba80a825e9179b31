// CPU check of the block operands formed on the host threads, built and run by
// tests/test_cpu_operands.py: prints a hash of every launch's operands (the same
// for any number of threads) and the largest difference of a block's matrix from
// its gates' product in std::complex.
#include "tcplan.cpp"

#include <cstdio>
#include <random>

using namespace qg;
typedef std::complex<double> cd;

int main() {
    std::mt19937_64 rng(17);
    std::uniform_real_distribution<double> uni(0, 6.283185307179586);
    unsigned long long hash = 1469598103934665603ULL;
    double worst = 0.;
    for (int trial = 0; trial < 12; ++trial) {
        const int n = 13 + trial % 4;
        std::vector<PendingGate> gates(160);
        for (auto &g : gates) {
            std::vector<int> lanes(n);
            for (int i = 0; i < n; ++i) lanes[i] = i;
            std::shuffle(lanes.begin(), lanes.end(), rng);
            g.target = lanes[0];
            g.controls.assign(lanes.begin() + 1, lanes.begin() + 1 + rng() % 4);
            const double th = uni(rng), a = uni(rng), b = uni(rng);
            cd m[4] = {std::cos(th), -std::polar(std::sin(th), a), std::polar(std::sin(th), b),
                       std::polar(std::cos(th), a + b)};
            if (rng() % 4 == 0) m[0] = m[3] = 0., m[1] = m[2] = 1.;  // X
            else if (rng() % 3 == 0) m[0] = rng() % 2 ? 1. : std::polar(1., a), m[3] = std::polar(1., b), m[1] = m[2] = 0.;
            for (int k = 0; k < 4; ++k) {
                g.m.v[2 * k] = m[k].real();
                g.m.v[2 * k + 1] = m[k].imag();
            }
            g.diag = is_diag(g.m);
        }
        std::vector<const PendingGate *> rem;
        for (auto &g : gates) rem.push_back(&g);
        while (!rem.empty()) {
            unsigned long long S = plan_stage_lanes(rem, 7, 12, false, kMaxTensorStageGates);
            std::vector<const PendingGate *> take, keep;
            stage_take(rem, S, rem.size(), &take, &keep, false, kMaxTensorStageGates);
            for (int q = 0; q < n && __builtin_popcountll(S) < 12; ++q) S |= 1ULL << q;
            const TileLanes tl = tile_lanes_of(S, n);
            const TcOps ops = tc_ops(tc_blocks(take, tl), true);
            for (size_t b0 = 0; b0 < ops.size();) {
                const int nb = tc_ops_per_launch(ops, b0, kFP64);
                static TcStageDesc desc;
                size_t bytes = 0;
                for (int b = 0; b < nb; ++b) bytes += tc_op_bytes(ops[b0 + b], kFP64);
                std::vector<unsigned char> buf(bytes);
                tc_plan_launch(tl, n, ops, b0, nb, desc, buf.data(), kFP64);
                auto mix = [&](const void *p, size_t k) {
                    for (size_t i = 0; i < k; ++i)
                        hash = (hash ^ ((const unsigned char *)p)[i]) * 1099511628211ULL;
                };
                mix(buf.data(), bytes);
                mix(desc.op_exp, sizeof(desc.op_exp));
                mix(desc.op_low, sizeof(desc.op_low));
                b0 += nb;
            }
            for (const TcOp &op : ops) {
                if (op.phase) continue;
                TcLayout lay;
                int k = 0;
                for (int p = 0; p < 12 && k < 5; ++p)
                    if (op.lanes >> p & 1u) lay.amps[k++] = p;
                for (int p = 0; p < 12 && k < 5; ++p)
                    if (!(op.lanes >> p & 1u)) lay.amps[k++] = p;
                cd U[1024], W[1024];
                tc_block_matrix(op.gates, tl, lay, U);
                int bit_of[64];
                for (int x = 0; x < 5; ++x) bit_of[lay.amps[x]] = x;
                for (int i = 0; i < 1024; ++i) W[i] = i / 32 == i % 32 ? 1. : 0.;
                for (auto *g : op.gates) {
                    const int tb = 1 << bit_of[tl.local_of[g->target]];
                    int cm = 0;
                    for (int c : g->controls) cm |= 1 << bit_of[tl.local_of[c]];
                    const double *v = g->m.v;
                    for (int r = 0; r < 32; ++r) {
                        if ((r & tb) || (r & cm) != cm) continue;
                        for (int c = 0; c < 32; ++c) {
                            const cd x = W[r * 32 + c], y = W[(r | tb) * 32 + c];
                            W[r * 32 + c] = cd(v[0], v[1]) * x + cd(v[2], v[3]) * y;
                            W[(r | tb) * 32 + c] = cd(v[4], v[5]) * x + cd(v[6], v[7]) * y;
                        }
                    }
                }
                for (int i = 0; i < 1024; ++i) worst = std::max(worst, std::abs(U[i] - W[i]));
            }
            rem.swap(keep);
        }
    }
    printf("hash %llu\nworst %.3e\n", hash, worst);
    return 0;
}
