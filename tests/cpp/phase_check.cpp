// CPU check of the complex128 tensor stage's phase ops: tables of tc_plan_launch,
// multiplied as phase_mul of qgate_gb300/csrc/dstage.cu does it, 32-bit negations
// included, against long double.  The phases' parts lie on and beside the ties
// of the table's two roundings.  Built and run by tests/test_cpu_phase_tables.py;
// prints "worst <error in units of V>" and "most <largest |low word|>".
#include "tcplan.cpp"

#include <cstdio>
#include <random>

using namespace qg;
typedef unsigned long long u64;

static int neg32(int x) { return (int)(0u - (unsigned)x); }  // wraps, as the GPU's does

int main() {
    std::mt19937_64 rng(11);
    const int n = 12;
    const TileLanes tl = tile_lanes_of((1ULL << n) - 1, n);
    double worst = 0, most = 0;
    const double fixed[] = {1.5, -1.5, 0.5, -0.5, 2.5, -2.5, 1.5 + 0x1p-22, 1.5 - 0x1p-22, 0.25};
    for (int k = 0; k < 400; ++k) {
        double s;
        if (k < 9) s = fixed[k] * 0x1p-30;
        else s = std::sin((double)(rng() >> 11) * 0x1p-53 * 6.283185307179586);
        if (k >= 9 && k % 3 == 0) s = ((double)(long long)(s * 0x1p29) + 0.5) * 0x1p-30;  // ties
        const double c = std::sqrt(1. - s * s) * (k & 1 ? -1. : 1.);
        const double entry[2][2] = {{c, s}, {s, c}};  // either part on the tie
        for (int swap = 0; swap < 2; ++swap) {
            PendingGate g;
            g.target = k % n;
            const double v[8] = {1, 0, 0, 0, 0, 0, entry[swap][0], entry[swap][1]};
            memcpy(g.m.v, v, sizeof(v));
            g.diag = true;
            const std::vector<const PendingGate *> gates{&g};
            const TcOps ops = tc_ops(tc_blocks(gates, tl), true);
            static TcStageDesc desc;
            std::vector<int> buf(tc_op_bytes(ops[0], kFP64) / 4);
            tc_plan_launch(tl, n, ops, 0, 1, desc, (unsigned char *)buf.data(), kFP64);
            const int *p = buf.data() + buf.size() - 4;  // the gate's lane set
            for (int j = 0; j < 4; j += 1) most = std::max(most, std::fabs((double)p[j] * (j & 1)));
            for (int t = 0; t < 8; ++t) {
                const long long re = (long long)(rng() >> 11) - (1ll << 52);
                const long long im = (long long)(rng() >> 11) - (1ll << 52);
                const long long rl = (int)(unsigned)re, il = (int)(unsigned)im;
                const long long rh = (re - rl) >> 32, ih = (im - il) >> 32;
                const long long half = 1ll << 29;
                const long long x = ((rh * p[0] + ih * neg32(p[2])) * 4) +
                                    ((rl * p[0] + il * neg32(p[2]) + rh * p[1] +
                                      ih * neg32(p[3]) + half) >> 30);
                const long long y = ((ih * p[0] + rh * p[2]) * 4) +
                                    ((il * p[0] + rl * p[2] + ih * p[1] + rh * p[3] + half) >> 30);
                const long double a = entry[swap][0], b = entry[swap][1];
                worst = std::max(worst, (double)std::fabs(x - (a * re - b * im)));
                worst = std::max(worst, (double)std::fabs(y - (a * im + b * re)));
            }
        }
    }
    printf("worst %.4f\nmost %.0f\n", worst, most);
    return 0;
}
