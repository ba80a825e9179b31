// CPU emulation of the complex128 tensor stage (qgate_gb300/csrc/dstage.cu) from
// launch plans of tcplan.cpp, in the kernel's own integer arithmetic: tile
// exponent, balanced digits, operand chunks, level sums, recombination, shift
// and the way back to FP64.  Built and run by tests/test_cpu_digits.py.  For
// every kind of state and matrix prints
//   <kind> <worst error / bound> <worst relative 2-norm error> <largest |level|>
// and the counts of structural faults.
#include "tcplan.cpp"

#include <cstdio>
#include <map>
#include <random>

using namespace qg;
typedef std::complex<double> cd;
typedef unsigned long long u64;

static const u64 kBias = 256ull | (512ull << 10) | (512ull << 20) | (512ull << 30) | (512ull << 40);
static int bad_digit = 0, bad_table = 0, direct_launches = 0, natural_launches = 0, phase_ops = 0;

static u64 bits_of(double x) {
    u64 b;
    memcpy(&b, &x, 8);
    return b;
}
static double of_bits(u64 b) {
    double x;
    memcpy(&x, &b, 8);
    return x;
}

static void digits_of(u64 w, double *dg) {  // w in eighths of the last digit; dg[0] = a1
    if (w >> 53) ++bad_digit;
    for (int k = 2; k < 5; ++k) dg[4 - k] = (double)((w >> (10 * k + 3)) & 1023u) - 512;
    dg[3] = 0.5 * (double)((w >> 12) & 2047u) - 512;
    dg[4] = 0.125 * (double)(w & 4095u) - 256;
}

static u64 biased_from_double(double x, int emax) {
    const u64 b = bits_of(x);
    const unsigned lo = (unsigned)b, hi = (unsigned)(b >> 32);
    const int e = (int)((hi >> 20) & 0x7ffu);
    const int s = std::min(e ? emax - e : 62, 62);
    const u64 m = ((u64)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    const u64 v = (m >> s) + 1ull;
    const u64 neg = (u64)((long long)(int)hi >> 31);
    return ((v >> 1) ^ neg) + (8 * kBias + (neg & 1ull));
}

static double double_from_fixed(long long V, int e) {
    const u64 sg = (u64)(V >> 63);
    const u64 u = ((u64)V ^ sg) + (sg & 1ull);
    if (u == 0) return 0.;
    const int lz = __builtin_clzll(u), eb = e + 1086 - lz;
    if (eb < 1) return 0.;
    return of_bits((((u64)(eb - 1) << 52) + ((u << lz) >> 11)) | (sg & (1ull << 63)));
}

int main() {
    std::mt19937 rng(77);
    std::normal_distribution<double> gauss(0, 1);
    std::uniform_real_distribution<double> uni(0, 6.283185307179586);
    const char *kinds[] = {"gaussian", "basis",  "uniform", "orders",    "hadamard", "tiny",
                           "single",   "shrink", "grow",    "projector", "qft",      "phases"};
    for (int kind = 0; kind < 12; ++kind) {
        const std::string K = kinds[kind];
        double worst_ratio = 0, worst_rel = 0;
        long long worst_level = 0;
        for (int trial = 0; trial < 6; ++trial) {
            const int n = 16;
            std::vector<PendingGate> gates;
            auto add = [&](int t, std::vector<int> c, cd a, cd b, cd cc, cd e) {
                PendingGate g;
                g.target = t;
                g.controls = c;
                const double v[8] = {a.real(), a.imag(), b.real(), b.imag(),
                                     cc.real(), cc.imag(), e.real(), e.imag()};
                memcpy(g.m.v, v, sizeof(v));
                g.diag = is_diag(g.m);
                gates.push_back(g);
            };
            if (K == "qft")  // H and the controlled phases below it, from the highest lane
                for (int i = n - 1; i >= 0; --i) {
                    const double r = std::sqrt(.5);
                    add(i, {}, r, r, r, -r);
                    for (int j = i - 1; j >= 0; --j)
                        add(i, {j}, 1, 0, 0, std::polar(1., 3.14159265358979323846 / (1 << (i - j))));
                }
            if (K == "phases")  // diagonal gates alone: one phase op
                for (int i = 0; i < 40; ++i)
                    add(i % n, {(i * 7 + 1 + trial) % n == i % n ? (i + 1) % n : (i * 7 + 1 + trial) % n},
                        std::polar(1., -uni(rng)), 0, 0, std::polar(1., uni(rng)));
            const int layers = K == "qft" || K == "phases" ? 0 : K == "single" ? 1 : 3;
            for (int l = 0; l < layers; ++l) {
                for (int q = 0; q < n; ++q) {
                    const double th = uni(rng), ph = uni(rng), la = uni(rng), r = std::sqrt(.5);
                    if (K == "single" && q != trial) continue;
                    if (K == "hadamard" || K == "uniform")
                        add(q, {}, r, r, r, -r);
                    else
                        add(q, {}, std::cos(th / 2), -std::polar(std::sin(th / 2), la),
                            std::polar(std::sin(th / 2), ph), std::polar(std::cos(th / 2), ph + la));
                    if (K == "shrink") add(q, {}, 1e-3, 0, 0, 3e-4);
                    if (K == "grow") add(q, {}, 700., 0, 0, -50.);
                    if (K == "projector" && q % 5 == 2) add(q, {}, 1, 0, 0, 0);
                }
                for (int q = 0; q + 1 < n && K != "single"; q += 2) {
                    const int c = (q + 3 * l + trial) % n, t = (q + 1 + 5 * l) % n;
                    if (c != t) add(t, {c}, 0, 1, 1, 0);
                }
            }
            std::vector<const PendingGate *> rem;
            for (auto &g : gates) rem.push_back(&g);
            const u64 S0 = plan_stage_lanes(rem, 7, 12, false, kMaxTensorStageGates);
            std::vector<const PendingGate *> take, keep;
            stage_take(rem, S0, rem.size(), &take, &keep, false, kMaxTensorStageGates);
            u64 S = S0;
            for (int q = 0; q < n && __builtin_popcountll(S) < 12; ++q) S |= 1ULL << q;
            const TileLanes tl = tile_lanes_of(S, n);
            const bool phases = K == "qft" || K == "phases";
            const TcOps ops = tc_ops(tc_blocks(take, tl), phases);
            const int nb = tc_ops_per_launch(ops, 0, kFP64);
            static TcStageDesc desc;
            size_t bytes = 0;
            for (const TcOp &op : ops) bytes += tc_op_bytes(op, kFP64);
            std::vector<unsigned char> buf(bytes);
            tc_plan_launch(tl, n, ops, 0, nb, desc, buf.data(), kFP64);
            if (desc.ops_bytes != buf.size() || (size_t)nb != ops.size()) ++bad_table;
            auto slot_of = [&](const SetSlots &ss, unsigned r, unsigned j) {
                unsigned slot = (unsigned)ss.lo[r & 31u] ^ (unsigned)ss.hi[r >> 5];
                for (int k = 0; k < 5; ++k)
                    if (j >> k & 1u) slot ^= ss.q[k];
                return slot;
            };
            for (int b = 0; b < nb + 2; ++b) {
                if (b < nb && desc.op_kind[b] == 1) {
                    ++phase_ops;
                    for (unsigned r = 0; r < 128; ++r)
                        for (unsigned j = 0; j < 32; ++j)
                            if (desc.op_off[b] + 16 * (slot_of(desc.sets[b], r, j) + 1) > bytes) ++bad_table;
                    continue;
                }
                std::vector<int> seen(4096, 0);
                for (unsigned r = 0; r < 128; ++r)
                    for (unsigned j = 0; j < 32; ++j) {
                        const unsigned sl = slot_of(desc.sets[b], r, j);
                        if (sl >= 4096 || seen[sl]++) ++bad_table;
                    }
            }
            auto offset = [&](const int *lane, const long long *e, unsigned r, unsigned j) {
                long long o = 0;
                for (int b = 0; b < 7; ++b)
                    if (r >> b & 1u) o |= 1LL << lane[b];
                for (int k = 0; k < 5; ++k)
                    if (j >> k & 1u) o += e[k];
                return o;
            };
            // the tile's state
            std::map<long long, cd> want, got;
            std::vector<std::vector<cd>> in(128, std::vector<cd>(32));
            double scale = K == "tiny" ? 1e-290 : 1.;
            for (unsigned r = 0; r < 128; ++r)
                for (unsigned j = 0; j < 32; ++j) {
                    cd x(gauss(rng), gauss(rng));
                    if (K == "basis") x = (r == 5 && j == 7) ? cd(0.6, 0.8) : cd(0, 0);
                    if (K == "uniform") x = cd(1. / 64, 0);
                    if (K == "orders") x *= std::pow(10., -(double)(rng() % 18));
                    in[r][j] = x * scale;
                    want[offset(desc.row_lane, desc.in_e, r, j)] = in[r][j];
                }
            if (want.size() != 4096) ++bad_table;
            double maxc = 0, norm = 0;
            for (auto &kv : want) {
                maxc = std::max(maxc, std::max(std::fabs(kv.second.real()), std::fabs(kv.second.imag())));
                norm += std::norm(kv.second / scale);
            }
            norm = std::sqrt(norm) * scale;
            // the kernel
            const unsigned mx = (unsigned)(bits_of(maxc) >> 32);
            const int emax = (int)((mx + 0x8000u) >> 20);
            int E = emax - 1071;
            std::vector<std::vector<u64>> W(4096, std::vector<u64>(2));
            std::vector<std::vector<long long>> V(128, std::vector<long long>(64));
            const bool first_phase = desc.op_kind[0] == 1;
            for (unsigned r = 0; r < 128; ++r)
                for (unsigned j = 0; j < 32; ++j) {
                    const double x = in[r][j].real(), y = in[r][j].imag();
                    if (first_phase) {
                        V[r][2 * j] = (long long)(biased_from_double(x, emax) - 8 * kBias);
                        V[r][2 * j + 1] = (long long)(biased_from_double(y, emax) - 8 * kBias);
                    } else {
                        W[slot_of(desc.sets[0], r, j)] = {biased_from_double(x, emax),
                                                          biased_from_double(y, emax)};
                    }
                }
            if (first_phase) E -= 3;
            double amp = 1.;  // what the blocks may enlarge the norm by (2^op_exp each)
            for (int b = 0; b < nb; ++b) {
                if (desc.op_kind[b] == 1) {
                    const int *tab = (const int *)(buf.data() + desc.op_off[b]);
                    for (unsigned r = 0; r < 128; ++r)
                        for (unsigned j = 0; j < 32; ++j) {
                            const int *p = tab + 4 * slot_of(desc.sets[b], r, j);
                            const long long re = V[r][2 * j], im = V[r][2 * j + 1];
                            const long long rl = (int)(unsigned)re, il = (int)(unsigned)im;
                            const long long rh = (re - rl) >> 32, ih = (im - il) >> 32;
                            const long long half = 1ll << 29;
                            V[r][2 * j] = ((rh * p[0] - ih * p[2]) << 2) +
                                          ((rl * p[0] - il * p[2] + rh * p[1] - ih * p[3] + half) >> 30);
                            V[r][2 * j + 1] =
                                ((ih * p[0] + rh * p[2]) << 2) +
                                ((il * p[0] + rl * p[2] + ih * p[1] + rh * p[3] + half) >> 30);
                        }
                    continue;
                }
                if (b > 0) {  // the integers' digits for this op
                    u64 top = 0;
                    for (auto &row : V)
                        for (long long x : row) {
                            const int hi = (int)(x >> 32);
                            top = std::max(top, (u64)(unsigned)(hi ^ (hi >> 31)));
                        }
                    const unsigned t32 = (unsigned)top + ((unsigned)top >> 5) + 1u;
                    const int sh = 15 - __builtin_clz(t32);
                    if (sh > 11) ++bad_digit;  // the kernel's field shifts stay below 32
                    E += sh;
                    for (unsigned r = 0; r < 128; ++r)
                        for (unsigned j = 0; j < 32; ++j) {
                            std::vector<u64> w(2);
                            for (int p = 0; p < 2; ++p) {
                                u64 x = (u64)V[r][2 * j + p];
                                if (sh < 3) x <<= 3 - sh;
                                const int rs = sh > 3 ? sh : 3;
                                w[p] = (x + (kBias << rs) + ((1ull << rs) >> 4)) >> (rs - 3);
                            }
                            W[slot_of(desc.sets[b], r, j)] = w;
                        }
                }
                const unsigned short *B = (const unsigned short *)(buf.data() + desc.op_off[b]);
                for (unsigned row = 0; row < 128; ++row) {
                    double a[5][64];
                    for (unsigned i = 0; i < 32; ++i) {
                        const unsigned c = (row << 5) | i;
                        const unsigned cs = c ^ (((c >> 5) & 7u) << 2);
                        for (int p = 0; p < 2; ++p) {
                            double dg[5];
                            digits_of(W[cs][p], dg);
                            for (int k = 0; k < 5; ++k) a[k][2 * i + p] = dg[k];
                        }
                    }
                    for (int o = 0; o < 64; ++o) {
                        double L[6] = {0, 0, 0, 0, 0, 0};
                        for (int j = 0; j < 5; ++j)
                            for (int k = 0; k < 64; ++k) {
                                const size_t at = (size_t)(4 * (o >> 5) + (k >> 4)) * 2560 +
                                                  (k % 16 / 8) * 1280 + (32 * j + (o & 31)) / 8 * 64 +
                                                  (32 * j + (o & 31)) % 8 * 8 + k % 8;
                                const double bv = f16_value(B[at]);
                                for (int i = 0; i < 5 && i + j <= 5; ++i) L[i + j] += a[i][k] * bv;
                            }
                        for (double x : L) worst_level = std::max(worst_level, (long long)std::fabs(x));
                        const float g = std::fmaf((float)L[5], 0x1p-10f, (float)L[4]);
                        V[row][o] = (long long)L[0] * (1ll << 34) + (long long)L[1] * (1ll << 24) +
                                    (long long)L[2] * (1ll << 14) + std::llrint(L[3] * 16) +
                                    std::llrint((double)g * 0x1p-6);
                    }
                }
                E += desc.op_exp[b] - 4;
                amp *= std::ldexp(1., std::max(0, (int)desc.op_exp[b]));
            }
            std::vector<std::vector<cd>> fin(128, std::vector<cd>(32));
            for (unsigned r = 0; r < 128; ++r)
                for (unsigned j = 0; j < 32; ++j)
                    fin[r][j] = cd(double_from_fixed(V[r][2 * j], E), double_from_fixed(V[r][2 * j + 1], E));
            if (desc.direct_out) {
                ++direct_launches;
                unsigned low = 0;
                for (int b = 0; b < 5; ++b) low |= 1u << desc.out_row_lane[b];
                if ((low & 7u) != 7u) ++bad_table;
                for (unsigned r = 0; r < 128; ++r)
                    for (unsigned j = 0; j < 32; ++j)
                        got[offset(desc.out_row_lane, desc.out_e, r, j)] = fin[r][j];
            } else {
                ++natural_launches;
                std::vector<cd> nat(4096);
                for (unsigned r = 0; r < 128; ++r)
                    for (unsigned j = 0; j < 32; ++j) nat[slot_of(desc.sets[nb], r, j)] = fin[r][j];
                for (unsigned r = 0; r < 128; ++r)
                    for (unsigned j = 0; j < 32; ++j)
                        got[offset(desc.row_lane, desc.in_e, r, j)] = nat[slot_of(desc.sets[nb + 1], r, j)];
            }
            // the gates themselves
            for (auto *g : take) {
                const long long tb = 1LL << g->target;
                long long cm = 0;
                for (int c : g->controls) cm |= 1LL << c;
                const cd m00(g->m.v[0], g->m.v[1]), m01(g->m.v[2], g->m.v[3]),
                    m10(g->m.v[4], g->m.v[5]), m11(g->m.v[6], g->m.v[7]);
                for (auto &kv : want) {
                    const long long off = kv.first;
                    if ((off & tb) || (off & cm) != cm) continue;
                    const cd a0 = want[off], a1 = want[off | tb];
                    want[off] = m00 * a0 + m01 * a1;
                    want[off | tb] = m10 * a0 + m11 * a1;
                }
            }
            if (got.size() != want.size()) ++bad_table;
            double err = 0, out = 0;
            for (auto &kv : want) {
                err += std::norm((got[kv.first] - kv.second) / scale);
                out += std::norm(kv.second / scale);
            }
            err = std::sqrt(err) * scale;
            out = std::sqrt(out) * scale;
            // Bound of the 2-norm error.  Per block and component: a rounded
            // digit tail of V is off by half a unit, at most 2^-52 of the
            // tile's largest component, 64 of them against a row of norm 1 give
            // 2^-49; matrix tails of 2^-53 against 64 components give 2^-47;
            // levels >= 8 less than 2^-52: together below 2^-46 of the largest
            // component, which never exceeds the tile's norm; over 8192
            // components 2^-39.5 of the norm in the worst case.
            const double bound = nb * std::ldexp(1., -39) * norm * amp;
            worst_ratio = std::max(worst_ratio, err / bound);
            if (out > 0) worst_rel = std::max(worst_rel, err / out);
        }
        printf("%s %.3e %.3e %lld\n", kinds[kind], worst_ratio, worst_rel, worst_level);
    }
    printf("bad_digit %d\nbad_table %d\ndirect %d\nnatural %d\nphase_ops %d\n", bad_digit, bad_table,
           direct_launches, natural_launches, phase_ops);
    return 0;
}
