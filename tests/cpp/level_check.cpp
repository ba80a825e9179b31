// CPU emulation of one dense op of the complex128 tensor stage (k_dstage) with
// FP32 accumulators that drop the bits below 2^-23 of a sum at every product of
// sixteen terms, in the kernel's order.  Tiles of (nearly) equal amplitudes under
// Hadamard blocks with a phase add all their digits in phase, which is what the
// accumulators have to hold.  Built and run by tests/test_cpu_levels.py; prints
// "<form> <worst relative error> <largest |accumulator|>" for the form the kernel
// uses (the products A2 B2 apart, smaller inputs for the ops that need them) and for
// one set of accumulators per level, the largest accumulator bound of any operand,
// and how many ops need smaller inputs.
#include "tcplan.cpp"

#include <cstdio>
#include <random>

using namespace qg;
typedef std::complex<double> cd;
typedef unsigned long long u64;

// One accumulation: the sum with the bits below its leading 24 cut off.
static double accumulate(double d, double x) {
    const double s = d + x;
    if (s == 0.) return 0.;
    int e;
    std::frexp(s, &e);
    const double u = std::ldexp(1., e - 24);
    return std::trunc(s / u) * u;
}

static double digit_b(const unsigned short *B, int j, int k, int o) {
    const size_t at = (size_t)(4 * (o >> 5) + (k >> 4)) * 2560 + (k % 16 / 8) * 1280 +
                      (32 * j + (o & 31)) / 8 * 64 + (32 * j + (o & 31)) % 8 * 8 + k % 8;
    return f16_value(B[at]);
}

int main() {
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> uni(0, 1);
    double worst[2] = {0, 0}, most[2] = {0, 0}, bound = 0;
    int lows = 0;
    std::vector<unsigned short> B(kDigitOpBytes / 2);
    for (int trial = 0; trial < 3000; ++trial) {
        // e^{i phi} H^{(x)5}, every second one with both parts' second digits near
        // their largest
        double phi;
        for (;;) {
            phi = uni(rng) * 6.283185307179586;
            const double re = std::cos(phi) * 32 * std::sqrt(32.), im = std::sin(phi) * 32 * std::sqrt(32.);
            if (trial % 2 || std::min(std::fabs(re - std::nearbyint(re)),
                                      std::fabs(im - std::nearbyint(im))) > 0.49)
                break;
        }
        cd U[1024];
        for (int o = 0; o < 32; ++o)
            for (int i = 0; i < 32; ++i)
                U[o * 32 + i] = std::polar(1. / std::sqrt(32.), phi) *
                                (double)(__builtin_popcount(o & i) & 1 ? -1 : 1);
        const bool low = tc_digit_rows(U, tc_digit_exponent(U), B.data());
        lows += low;
        for (int o = 0; o < 64; ++o) {
            double n1[3] = {0, 0, 0}, n2 = 0;  // 1-norms of B1..B3, 2-norm of B1
            for (int k = 0; k < 64; ++k) {
                for (int j = 0; j < 3; ++j) n1[j] += std::fabs(digit_b(B.data(), j, k, o));
                n2 += digit_b(B.data(), 0, k, o) * digit_b(B.data(), 0, k, o);
            }
            n2 = std::sqrt(n2);
            // A1 within 498 (249 for low ops), the others within 512, 64 of each
            const double a1 = low ? 249. : 498.;
            bound = std::max(bound, 8. * a1 * n2);                 // A1 B1
            bound = std::max(bound, a1 * n1[1] + 4096. * n2);      // A1 B2 + A2 B1
            bound = std::max(bound, a1 * n1[2] + 4096. * n2);      // A1 B3 + A3 B1
            bound = std::max(bound, 512. * n1[1]);                 // A2 B2
        }
        // a row of amplitudes whose mantissas are alike
        const double mr = trial % 2 ? 1. + uni(rng) * 0.94 : 1.9 + 0.04 * uni(rng), mi = mr;
        const double spread = trial % 8 < 2 ? 0. : 1e-4;
        double a[64];
        for (int i = 0; i < 32; ++i) {
            const double s = (trial % 7 == 2 && (i & 4)) ? -1. : 1.;
            a[2 * i] = s * mr * (1. + spread * (uni(rng) - .5));
            a[2 * i + 1] = -s * mi * (1. + spread * (uni(rng) - .5)) * (trial % 5 == 4 ? -1. : 1.);
        }
        for (int form = 0; form < 2; ++form) {  // 0: the kernel's, 1: one set per level
            const int top = form == 0 && low ? 48 : 49;
            double dg[5][64];
            for (int k = 0; k < 64; ++k) {
                double x = a[k] * 0.5;  // below 2^top after scaling: digits of radix 2^10
                x = std::ldexp(x, top - 40);
                for (int j = 0; j < 5; ++j) {
                    dg[j][k] = j < 3 ? std::nearbyint(x)
                                     : j == 3 ? std::nearbyint(x * 2) / 2 : std::nearbyint(x * 8) / 8;
                    x = (x - dg[j][k]) * 1024.;
                }
            }
            double err = 0, ref = 0;
            for (int o = 0; o < 64; ++o) {
                double L[7] = {0, 0, 0, 0, 0, 0, 0};
                for (int ks = 0; ks < 4; ++ks)
                    for (int i = 0; i < 5; ++i)
                        for (int j = 0; i + j <= 5 && j < 5; ++j) {
                            double s = 0;
                            for (int k = 16 * ks; k < 16 * ks + 16; ++k)
                                s += dg[i][k] * digit_b(B.data(), j, k, o);
                            double &acc = form == 0 && i == 1 && j == 1 ? L[6] : L[i + j];
                            acc = accumulate(acc, s);
                            if (i + j <= 2) most[form] = std::max(most[form], std::fabs(acc));
                        }
                long double v = 0;
                for (int l = 0; l < 6; ++l)
                    v += (long double)(L[l] + (l == 2 ? L[6] : 0.)) * std::ldexp(1.L, -10 * l);
                v = std::ldexp(v, 31 - top);  // (b1: 2^10, a1: 2^(top - 40), halved inputs)
                long double want = 0;
                for (int i = 0; i < 32; ++i) {
                    const cd u = U[(o >> 1) * 32 + i];
                    want += (o & 1) ? (long double)u.imag() * a[2 * i] + (long double)u.real() * a[2 * i + 1]
                                    : (long double)u.real() * a[2 * i] - (long double)u.imag() * a[2 * i + 1];
                }
                err += (double)((v - want) * (v - want));
                ref += (double)(want * want);
            }
            worst[form] = std::max(worst[form], std::sqrt(err / ref));
        }
    }
    printf("kernel %.3e %.0f\nper_level %.3e %.0f\nbound %.0f 0\nlows %d 0\n", worst[0], most[0], worst[1], most[1],
           bound, lows);
    return 0;
}
