// Tensor-core stage kernel for complex128 states (k_dstage).
//
// A tile of 12 lanes (4096 amplitudes, 64 KB) stays on chip while a sequence
// of fused 5-lane blocks, each a 32x32 complex unitary, is applied to it.  As
// in the complex64 stage (tcstage.cu) a block is D[128 x 64] = A[128 x 64]
// B[64 x 64] in real form, but FP64 accuracy comes from error-free products
// of digit slices on the FP16 tensor pipe (the splitting of Ozaki, Ogita,
// Oishi and Rump, "Error-free transformations of matrix multiplication by
// using fast routines of matrix multiplication", 2012):
//
//  - the tile is held as 64-bit integers V with one exponent per tile; before
//    a block V is shifted so that |V| < 0.97 2^49 and cut into five balanced
//    radix-2^10 digits a1..a5 (|a1| <= 498, |a| <= 512, a4 in halves, a5 within
//    256 in eighths: exact in FP16);
//  - the host cuts every entry of the block's matrix, scaled so that its rows
//    have norm <= 1, into digits b1 (|b1| <= 1024), b2..b5 (|b| <= 512; b5 in
//    quarters);
//  - level L_d = sum over i + j = d of A_i B_j, d = 2..7, accumulates in its
//    own FP32 columns of tensor memory, A_2 B_2 in a seventh set.  The sums of
//    d <= 4 are integers that FP32 holds exactly, whatever the tile: of 64 terms
//    each, with ||B_1|| <= 2^10 + 4 (2-norm of a column), |A_1 B_1| <= 2^22 and
//    |A_2 B_2| <= 2^24; |A_1 B_j + A_j B_1| <= 498 |B_j|_1 + 2^12 (2^10 + 4), j = 2, 3,
//    stays below 2^24 where B_2's and B_3's columns have 1-norms of at most 3/4 of
//    their largest 2^15 (a block of random entries has about 2^14).  The host
//    finds the ops where they are larger (op_low): before those V is shifted one
//    bit further, |a1| <= 249.  (With one set per level, a Hadamard block with a
//    phase on a tile of equal amplitudes, whose digits all add up, went past 2^24
//    at level 4, for some phases at level 3 too: errors up to 4.9e-10.)
//    L_5 may pass 2^24, and then rounds at 2^-52 of the row's norm;
//  - the result sum_d L_d 2^(-10 (d - 2)) is formed as a 64-bit integer again.
// What is left out: digits of V below 2^-52 of the tile's largest component
// (rounded), of the matrix below 2^-53, and levels d >= 8 (2^-60).  These are errors of
// the size of the tile's largest amplitude, where double-float arithmetic errs by the
// size of what a gate combines.  So a tile is stored only if its smallest
// amplitude lies within 2^16 of the largest that its last block read, and is right
// to 2^-35 of each amplitude then.  Any other tile (products of small rotations, exact
// zeros, which may stand for less than a digit, rare outcomes beside common ones)
// is left as it was and marked, and the same gates run on it on the CUDA cores
// (k_rstage_marked).  16: mixed states hold next to no such tile (random U3 + CX, 22
// lanes, from the third pass on: none of 10^4; with 13, one in 10^3), while a QFT
// of a product state has them in half of its passes.  Finding them costs nothing
// that can be measured; a launch of k_rstage_marked that has none takes 8 us.  A tile
// that holds an amplitude (not zero) 2^20 below its largest when it is loaded is left
// at once: states of small rotations, 24 lanes, 3 passes, 4.8 ms without that, 3.75
// with it (3.17 on the CUDA cores alone).
// Stages with a matrix that is not unitary do not come here (products of such
// matrices can have rows of very different norm), nor do those without a gate
// that mixes amplitudes: diagonal ones run as one FP64 table (k_phase_f64),
// permutations on the CUDA cores.
// Whole circuits against 64-bit arithmetic (2-norm): random U3 + CX, 26 qubits, 12
// layers 8.2e-15 (the double-float CUDA-core stages: 5.2e-14), a 25-qubit QFT of
// a product state 5.9e-15 (2.5e-14).
//
// Diagonal gates of one tile run as phase ops (see phase_mul): a table of 64-bit
// fixed-point phases multiplied into V.
//
// Data path.  Two groups of 256 threads (two threads per tile row, 16
// amplitudes each) work on a tile each; warp 16 issues the products of both, warp
// 17 streams the blocks' operands.  The products of a block run in two halves
// of 16 outputs (7 sets x 32 columns each): while the tensor core works on
// one half, the threads read the other back, and while one group cuts its
// tile into digits the other's products run.  Operands arrive in chunks of
// 10 KB (one half, two K-steps of 16) through a ring of three chunks per group.
//
// Bound: shared memory, then the groups' chain of phases.  Per tile and block the
// tensor core reads 230 KB of A and 156 KB of B, 40 KB of operands arrive and the
// threads write 80 KB of digits: 4000 cycles at 128 B per cycle, beside 2800 of
// products (19 of the 25 digit pairs, 350 cycles per K-step) and about 2400
// issue slots per scheduler, half of them on the integer pipe.  Measured on the
// 26-qubit, 12-layer random circuit (3.06 blocks per pass): 17 passes of 1.1 ms,
// 6600 cycles per tile and block; the CUDA-core stages take 22 passes of 3.6 ms.
// A pass's HBM time is 0.32 ms.  Steps on the way: the products issued from one
// thread's branch 1.8 ms a pass (operand moves, 200 cycles each, not the products,
// were the limit), addresses formed bit by bit at every use and FP64 conversions
// with branches 1.7 ms, 5 KB operand chunks instead of 10 KB 1.2 ms.
//
// Every wait is bounded: the mbarrier waits by themselves, the polls of the issuing
// warp and of the operand thread by a count that starts again whenever a group
// takes a tile, so that it bounds a wait and not the launch.  One that gives up
// sets g_ds_status; a group decides as a whole whether it leaves (abort_sh[g],
// written before its barrier and read after it, by its own threads only), the
// issuing warp leaves when both have, and the CTA frees its tensor memory.
#include <algorithm>
#include <cstdint>

#include "qg_device.cuh"
#include "qg_internal.h"
#include "qg_regstage.cuh"
#include "qg_tc.cuh"

namespace qg {

__device__ StageStatus g_ds_status;

namespace {

constexpr unsigned kSlice = 16384u;                  // one digit slice of a tile
constexpr unsigned kGroupA = kDigits * kSlice;       // a tile's digits
constexpr unsigned kStep = kDigitChunkBytes;         // one K-step: 160 x 16 FP16 values
constexpr unsigned kChunk = 2 * kStep;               // what the ring holds: two K-steps
constexpr int kRing = 3;
constexpr unsigned kGT = 256u;                       // threads per group
// Two groups and one warpgroup of which warp 16's first thread works.  The
// launch gives 96 registers a thread (61440 in all); the issuing warpgroup
// returns 64 of its own, so that the groups hold 112: 512 x 112 + 128 x 32.
constexpr unsigned kThreads = 2u * kGT + 128u;
// A tile with an amplitude below 2^-16 of the largest input of its last block is left
// to the CUDA cores: that input is scaled to 2^49, the block's outputs are 2^4 larger, and
// these are the high words of 64 bits.
constexpr unsigned kLeast = 1u << (49 + 4 - 16 - 32);
// (Only where the largest lies in [2^-45, 2^100): the CUDA cores' FP32 pairs have
// FP32's exponents, and err by up to 2^-97 below 2^-74.)
constexpr int kRangeLow = 1023 - 45, kRangeHigh = 1023 + 100;
// A loaded tile with an amplitude (not zero) this far below its largest is left to
// them at once.
constexpr unsigned kSkipBits = 20;
constexpr unsigned kLevelCols = 32u, kHalfCols = 7u * kLevelCols;

// Balanced digits: adding 512 to each of the five (256 to the last) makes them
// unsigned fields.
constexpr unsigned long long kBias = 256ull | (512ull << 10) | (512ull << 20) | (512ull << 30) |
                                     (512ull << 40);

__device__ __forceinline__ void tmem_ld_x4(unsigned taddr, unsigned (&u)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3])
                 : "r"(taddr));
}

__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Fields of two numbers (re, im) at the low 10 bits of x and y as digits in
// FP16 (re low): 0x6400 | f is 1024 + f, and 1536 = 1024 + 512.
__device__ __forceinline__ unsigned digit_pair(unsigned x, unsigned y, unsigned one) {
    unsigned p = __byte_perm(x, y, 0x5410);
    p = (p & 0x03ff03ffu) | one;  // one: 0x64006400, kept in a register
    unsigned r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(p), "r"(0x66006600u));
    return r;
}

// The fourth digits keep halves, the last ones, within +-256, eighths: FP16 has
// room for them, and every bit halves what a block's input loses.  Their fields
// are 11 and 12 bits (the bits below the tenth: 0x3c00 | h << k is 1 + h 2^(k - 10)).
__device__ __forceinline__ unsigned digit4_pair(unsigned x, unsigned y, unsigned one) {
    const unsigned p = __byte_perm(x, y, 0x5410);
    const unsigned w = ((p >> 1) & 0x03ff03ffu) | one;
    const unsigned h = ((p * 512u) & 0x02000200u) | 0x3c003c00u;
    unsigned r;
    asm("{\n\t.reg .b32 t;\n\tsub.rn.f16x2 t, %1, %2;\n\tadd.rn.f16x2 %0, t, %3;\n\t}\n"
        : "=r"(r)
        : "r"(w), "r"(0x66016601u), "r"(h));  // 1537
    return r;
}
__device__ __forceinline__ unsigned digit5_pair(unsigned x, unsigned y, unsigned one) {
    const unsigned p = __byte_perm(x, y, 0x5410);
    const unsigned w = ((p >> 2) & 0x03ff03ffu) | one;
    const unsigned h = ((p * 128u) & 0x01800180u) | 0x3c003c00u;
    unsigned r;
    asm("{\n\t.reg .b32 t;\n\tfma.rn.f16x2 t, %1, %2, %3;\n\tadd.rn.f16x2 %0, t, %4;\n\t}\n"
        : "=r"(r)
        : "r"(w), "r"(0x38003800u), "r"(0xe202e202u), "r"(h));  // 1/2, -769
    return r;
}

// The five digits of (re, im), biased integers in units of 2^-sh, to the
// operand slot at shared address `at` of every slice; 3 <= sh <= 11.
__device__ __forceinline__ void put_digits(unsigned at, unsigned long long re,
                                           unsigned long long im, int sh, unsigned one) {
    const unsigned rl = (unsigned)re, rh = (unsigned)(re >> 32);
    const unsigned il = (unsigned)im, ih = (unsigned)(im >> 32);
    const unsigned d1 = digit_pair(rh >> (sh + 8), ih >> (sh + 8), one);
    const unsigned d2 = digit_pair(rh >> (sh - 2), ih >> (sh - 2), one);
    const unsigned d3 =
        digit_pair(__funnelshift_r(rl, rh, sh + 20), __funnelshift_r(il, ih, sh + 20), one);
    const unsigned d4 =
        digit4_pair(__funnelshift_r(rl, rh, sh + 9), __funnelshift_r(il, ih, sh + 9), one);
    const unsigned d5 =
        digit5_pair(__funnelshift_r(rl, rh, sh - 3), __funnelshift_r(il, ih, sh - 3), one);
    asm volatile(
        "st.shared.b32 [%0], %1;\n\t"
        "st.shared.b32 [%0 + 16384], %2;\n\t"
        "st.shared.b32 [%0 + 32768], %3;\n\t"
        "st.shared.b32 [%0 + 49152], %4;\n\t"
        "st.shared.b32 [%0 + 65536], %5;\n" ::"r"(at),
        "r"(d1), "r"(d2), "r"(d3), "r"(d4), "r"(d5)
        : "memory");
}

__device__ __forceinline__ unsigned long long join64(unsigned lo, unsigned hi) {
    return ((unsigned long long)hi << 32) | lo;
}

// What combine_levels leaves in its results.
constexpr unsigned kOffset = 0x4B400000u;

// FP64 bits -> biased integer in units of 2^(emax - 1074), an eighth of the
// last digit's, rounded to nearest; every exponent field is at most emax.
// Subnormals read as 0.
__device__ __forceinline__ unsigned long long biased_from_double(unsigned lo, unsigned hi, int emax) {
    const int e = (int)((hi >> 20) & 0x7ffu);
    const int s = min(e ? emax - e : 62, 62);
    const unsigned long long v = (join64(lo, (hi & 0xfffffu) | 0x100000u) >> s) + 1ull;  // twice
    const unsigned long long neg = (unsigned long long)((long long)(int)hi >> 31);
    return ((v >> 1) ^ neg) + (8ull * kBias + (neg & 1ull));
}

// (V - offset) * 2^e as FP64 bits (|V| < 2^58: at most five bits are cut
// off); below 2^-1022 reads as 0.
__device__ __forceinline__ void double_from_fixed(unsigned &lo, unsigned &hi, unsigned offset,
                                                  int e) {
    unsigned long long u = join64(lo, hi) - offset;
    const unsigned s = (unsigned)((int)(unsigned)(u >> 32) >> 31);
    u = (u ^ join64(s, s)) + (s & 1u);
    const unsigned h = (unsigned)(u >> 32);
    const int lz = __clz((int)(h ? h : (unsigned)u)) + (h ? 0 : 32);
    u <<= (lz & 63);
    const int eb = e + 1086 - lz;  // biased exponent of the leading bit
    const bool some = lz < 64 && eb >= 1;
    const unsigned m = (unsigned)(u >> 43) + ((unsigned)(eb - 1) << 20) + (s & 0x80000000u);
    lo = some ? (unsigned)(u >> 11) : 0u;
    hi = some ? (eb > 2046 ? 0x7ff00000u | (s & 0x80000000u) : m) : 0u;
}

// a * b + c in 64 bits.
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

// kOffset + sum_d L_d 2^(34 - 10 (d - 2)) of the six levels, |sum| < 2^57; u4b is
// A_2 B_2.  L_3..L_5 become integers by conversion; L_2 and, summed in FP32
// first (their rounding lies 2^-24 below L_6), L_6 and L_7 by the 1.5 * 2^23
// addition, whose bits 0x4B400000 stay in the low word (kOffset; it makes that
// word positive, so no sign is extended) and are taken out of the high word by
// its start value.  The multipliers come in registers: a multiply-add of 64
// bits is one instruction off the integer pipe, which bounds the kernel's
// arithmetic, where shifts and adds of 64 bits are four on it.
__device__ __forceinline__ void combine_levels(unsigned u2, unsigned u3, unsigned u4, unsigned u5,
                                               unsigned u6, unsigned u7, unsigned u4b, int m14,
                                               int m24, unsigned &lo, unsigned &hi) {
    constexpr float kMagic = 12582912.f;  // bits 0x4B400000
    const int i3 = __float2int_rn(__uint_as_float(u3));
    const int i4 = __float2int_rn(__uint_as_float(u4)) + __float2int_rn(__uint_as_float(u4b));
    const unsigned b2 = __float_as_uint(__fadd_rn(__uint_as_float(u2), kMagic));
    const float g = __fmaf_rn(__uint_as_float(u7), 0x1p-10f, __uint_as_float(u6));
    const unsigned t = (unsigned)__float2int_rn(__uint_as_float(u5) * 16.f) +
                       __float_as_uint(__fmaf_rn(g, 0x1p-6f, kMagic));
    const long long start =
        (long long)(((unsigned long long)(0u - kOffset * 4u) << 32) | t);
    const long long acc = mad_wide(i3, m24, mad_wide(i4, m14, start));
    lo = (unsigned)acc;
    hi = (unsigned)((unsigned long long)acc >> 32) + b2 * 4u;
}

// (re, im) - offset times the phase p = (x + y 2^-32, z + w 2^-32) 2^-30, rounded;
// the products of two low words are dropped (each below one unit, a quarter
// on average).  y and w lie within +-(2^31 - 1), as w is negated here.
__device__ __forceinline__ void phase_mul(unsigned (&v)[64], int j, unsigned offset, int4 p) {
    const unsigned long long re = join64(v[4 * j], v[4 * j + 1]) - offset;
    const unsigned long long im = join64(v[4 * j + 2], v[4 * j + 3]) - offset;
    const int rl = (int)(unsigned)re, il = (int)(unsigned)im;  // signed low words
    const int rh = (int)(unsigned)(re >> 32) + (int)((unsigned)re >> 31);
    const int ih = (int)(unsigned)(im >> 32) + (int)((unsigned)im >> 31);
    const long long a = mad_wide(rh, p.x, mad_wide(ih, -p.z, 0));
    const long long b = mad_wide(ih, p.x, mad_wide(rh, p.z, 0));
    const long long half = 1ll << 29;
    const long long c =
        mad_wide(rl, p.x, mad_wide(il, -p.z, mad_wide(rh, p.y, mad_wide(ih, -p.w, half))));
    const long long e =
        mad_wide(il, p.x, mad_wide(rl, p.z, mad_wide(ih, p.y, mad_wide(rh, p.w, half))));
    const unsigned long long x = (unsigned long long)((a << 2) + (c >> 30));
    const unsigned long long y = (unsigned long long)((b << 2) + (e >> 30));
    v[4 * j] = (unsigned)x;
    v[4 * j + 1] = (unsigned)(x >> 32);
    v[4 * j + 2] = (unsigned)y;
    v[4 * j + 3] = (unsigned)(y >> 32);
}

// Parameters of a group's walk over its 16 registers: register bits 0..2 are
// the layout's amplitude bits 0..2, register bit 3 its bit 4; the thread's half
// (hh) is bit 3, as the read-back of the products' halves leaves them.
template <class F> __device__ __forceinline__ void slots_walk(const SetSlots &ss, unsigned r,
                                                              unsigned hh, F f) {
    unsigned slot = (unsigned)ss.lo[r & 31u] ^ (unsigned)ss.hi[r >> 5];
    if (hh) slot ^= ss.q[3];
    const unsigned q[4] = {ss.q[0], ss.q[1], ss.q[2], ss.q[4]};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int j = i ^ (i >> 1);
        if (i > 0) slot ^= q[gray_bit(i)];
        f(j, slot);
    }
}
template <class P, class F> __device__ __forceinline__ void lanes_walk(P *p, const long long *e,
                                                                       F f) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int j = i ^ (i >> 1);
        if (i > 0) {
            const int k = gray_bit(i);
            const long long o = e[k == 3 ? 4 : k];
            p = (j >> k & 1) ? p + o : p - o;
        }
        f(j, p);
    }
}

// PH: the launch has phase ops (without them the kernel keeps the registers of
// the dense path alone).
template <bool PH>
__global__ void __launch_bounds__(kThreads, 1)
k_dstage(uint4 *__restrict__ s, const __grid_constant__ TcStageDesc d, int tiles,
         const TileMarks marks) {
    extern __shared__ __align__(1024) unsigned char smraw[];
    unsigned char *ring = smraw + 2 * kGroupA;                 // [group][kRing] chunks
    SetSlots *sset = (SetSlots *)(ring + 2 * kRing * kChunk);
    __shared__ __align__(8) unsigned long long bar_a[2], bar_d[2][2], bar_dfree[2],
        bar_b[2][kRing], bar_e[2][kRing], bar_end;
    __shared__ unsigned tmem_sh;
    __shared__ unsigned red[2][2][8];
    __shared__ __align__(16) uint2 range_sh[2][2][8];  // a loaded tile's largest, smallest part
    __shared__ volatile int wide_sh[2];  // the last tile (+ 1) found wide
    __shared__ volatile int done_sh[2];
    __shared__ int abort_sh[2];
    __shared__ volatile unsigned beat_sh[2];  // tiles taken by each group
    __shared__ volatile int stop_sh;
    __shared__ long long row_off[2][40];
    __shared__ unsigned dense_op[kMaxTcBlocks];  // the dense op after op b, in a circle
    __shared__ int dense_0;                       // the first dense op (-1: none)
    const unsigned tid = threadIdx.x, warp = tid >> 5;
    const int nb = d.nblocks;

    if ((smem_u32(smraw) & 1023u) != 0u) {
        if (tid == 0) report_stage(&g_ds_status, 4u, 4u << 8);
        return;
    }
    if (tid == 0) stop_sh = *(volatile unsigned *)&g_ds_status.bits != 0u;
    __syncthreads();
    if (stop_sh) return;
    __syncthreads();
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_u32(&tmem_sh)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int g = 0; g < 2; ++g) {
            mbar_init(smem_u32(&bar_a[g]), 8);
            mbar_init(smem_u32(&bar_dfree[g]), 8);
            for (int h = 0; h < 2; ++h) mbar_init(smem_u32(&bar_d[g][h]), 1);
            for (int k = 0; k < kRing; ++k) {
                mbar_init(smem_u32(&bar_b[g][k]), 1);
                mbar_init(smem_u32(&bar_e[g][k]), 1);
            }
            done_sh[g] = 0;
            wide_sh[g] = 0;
            abort_sh[g] = 0;
            beat_sh[g] = 0u;
        }
        mbar_init(smem_u32(&bar_end), 1);
        mbar_fence_init();  // bulk copies and commits arrive through the async proxy
        stop_sh = 0;
        dense_0 = -1;
        for (int b = nb - 1; b >= 0; --b)
            if (d.op_kind[b] == 0) dense_0 = b;
        int to = dense_0;
        for (int b = nb - 1; b >= 0; --b) {
            dense_op[b] = (unsigned)to;
            if (d.op_kind[b] == 0) to = b;
        }
    }
    rs::copy_sets(sset, d.sets, nb + 2, tid, kThreads);
    // Row offsets of the load and the final layout: by the thread's lane (row
    // bits 0..4), then by its warp in the group (row bits 5, 6, half).
    if (tid < 80u) {
        const int f = tid >= 40u, i = (int)tid - 40 * f;
        const int *lane = f ? d.out_row_lane : d.row_lane;
        const long long half = f ? d.out_e[3] : d.in_e[3];
        long long o = 0;
        for (int b = 0; b < 5; ++b)
            if (i < 32 && (i >> b & 1)) o |= 1LL << lane[b];
        if (i >= 32) {
            if (i & 1) o |= 1LL << lane[5];
            if (i & 2) o |= 1LL << lane[6];
            if (i & 4) o |= half;
        }
        row_off[f][i] = o;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_sh;

    if (warp >= 16) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n" ::: "memory");
        // ---- products and operand stream of both groups (one thread)
        const unsigned ring0 = smem_u32(ring);
        if (tid == 2u * kGT + 32u) {
            // ---- operand stream: keeps both rings full
            unsigned loaded[2] = {0u, 0u}, slot[2] = {0u, 0u}, part[2] = {0u, 0u};
            unsigned op[2] = {(unsigned)dense_0, (unsigned)dense_0};
            unsigned par[2] = {1u, 1u};  // the first round's slots are free
            unsigned beat = 0u;
            for (unsigned idle = 0; idle < (1u << 22); ++idle) {
                if (stop_sh) break;
                if (beat_sh[0] + beat_sh[1] != beat) {
                    beat = beat_sh[0] + beat_sh[1];
                    idle = 0;
                }
                if (idle > 1u) __nanosleep(200);
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if (dense_0 < 0 || (int)(blockIdx.x + g * gridDim.x) >= tiles) continue;
                    if (!mbar_test(smem_u32(&bar_e[g][slot[g]]), par[g])) continue;
                    bulk_load(ring0 + ((unsigned)g * kRing + slot[g]) * kChunk,
                              d.bmats + d.op_off[op[g]] + part[g] * kChunk, kChunk,
                              smem_u32(&bar_b[g][slot[g]]));
                    idle = 0;
                    ++loaded[g];
                    if (++slot[g] == (unsigned)kRing) {
                        slot[g] = 0u;
                        par[g] ^= 1u;
                    }
                    if (++part[g] == 4u) {
                        part[g] = 0u;
                        op[g] = dense_op[op[g]];
                    }
                }
            }
#pragma unroll
            for (int g = 0; g < 2; ++g)  // copies in flight: the last kRing at most
                for (unsigned c = loaded[g] > (unsigned)kRing ? loaded[g] - kRing : 0u;
                     c < loaded[g]; ++c)
                    mbar_wait(smem_u32(&bar_b[g][c % (unsigned)kRing]),
                              (c / (unsigned)kRing) & 1u);
        } else if (warp == 16) {
            // ---- the products of both groups (the whole warp walks, one lane
            // issues)
            const unsigned lane = elect_lane();
            bool ok = true;
            int active = 0;
            for (int g = 0; g < 2; ++g)
                if ((int)(blockIdx.x + g * gridDim.x) < tiles) active |= 1 << g;
            unsigned slot[2] = {0u, 0u}, par[2] = {0u, 0u}, apar[2] = {0u, 0u};
            unsigned fpar = 1u;  // parity of the free-column waits: the first passes
            unsigned idle = 0, beat = 0u;
            // (one decision for the whole warp at every wait)
            auto all = [](bool x) { return __all_sync(0xffffffffu, x) != 0; };
            const uint64_t da0 = smem_desc(smem_u32(smraw), 16, 1024, 2);
            const uint64_t db0 = smem_desc(ring0, 2560, 128);
#pragma unroll 1
            while (active && ok) {
                if (!all(beat_sh[0] + beat_sh[1] == beat)) {
                    beat = beat_sh[0] + beat_sh[1];
                    idle = 0;
                }
                if (++idle > (1u << 23)) ok = false;
                if (idle > 1u) __nanosleep(40);
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if (!(active >> g & 1) || !ok) continue;
                    if (!all(mbar_test(smem_u32(&bar_a[g]), apar[g]))) continue;
                    idle = 0;
                    apar[g] ^= 1u;
                    if (all(done_sh[g] != 0)) {
                        active &= ~(1 << g);
                        continue;
                    }
#pragma unroll
                    for (unsigned h = 0; h < 2u; ++h) {
                        ok = ok && all(mbar_wait(smem_u32(&bar_dfree[h]), fpar));
                        const unsigned dcol = tmem + h * kHalfCols;
#pragma unroll
                        for (unsigned kp = 0; kp < 2u; ++kp) {
                            const unsigned k = slot[g];
                            ok = ok && all(mbar_wait(smem_u32(&bar_b[g][k]), par[g]));
                            if (!ok) break;
                            tc_fence_after();
                            // A_i: 128-byte swizzled K-major; B_1..: no
                            // swizzle, 160 rows, 8-row groups 128 bytes and
                            // 8-element K-groups 2560 bytes apart.  Level
                            // i + j: columns 32 (i + j - 2); A_2 B_2: columns
                            // 192 and up.
#pragma unroll
                            for (unsigned q = 0; q < 2u; ++q) {
                                const unsigned ks = 2u * kp + q;
                                const uint64_t db = db0 + (uint64_t)(((unsigned)g * kRing + k) *
                                                                     (kChunk >> 4)) +
                                                    q * (kStep >> 4);
                                // 32 bytes per K-step; kNext: the next slice
                                const uint64_t da = da0 + (uint64_t)g * (kGroupA >> 4) + 2u * ks;
                                constexpr uint64_t kNext = kSlice >> 4;
                                mma_f16_lane(dcol, da, db, ks > 0u ? 1u : 0u, idesc_f16(128, 160),
                                             lane);
                                constexpr uint64_t kB = 512u >> 4;  // 32 rows of B
                                mma_f16_lane(dcol + 32u, da + kNext, db, 1u, idesc_f16(128, 32),
                                             lane);
                                mma_f16_lane(dcol + 192u, da + kNext, db + kB, ks > 0u ? 1u : 0u,
                                             idesc_f16(128, 32), lane);
                                if (ks == 0u) {
                                    // level 7 is first written here
                                    mma_f16_lane(dcol + 96u, da + kNext, db + 2 * kB, 1u,
                                                 idesc_f16(128, 64), lane);
                                    mma_f16_lane(dcol + 160u, da + kNext, db + 4 * kB, 0u,
                                                 idesc_f16(128, 32), lane);
                                } else {
                                    mma_f16_lane(dcol + 96u, da + kNext, db + 2 * kB, 1u,
                                                 idesc_f16(128, 96), lane);
                                }
                                mma_f16_lane(dcol + 64u, da + 2 * kNext, db, 1u,
                                             idesc_f16(128, 128), lane);
                                mma_f16_lane(dcol + 96u, da + 3 * kNext, db, 1u, idesc_f16(128, 96),
                                             lane);
                                mma_f16_lane(dcol + 128u, da + 4 * kNext, db, 1u,
                                             idesc_f16(128, 64), lane);
                            }
                            if (lane) {
                                if (kp == 1u) mma_commit(smem_u32(&bar_d[g][h]));
                                mma_commit(smem_u32(&bar_e[g][k]));
                            }
                            __syncwarp();
                            if (++slot[g] == (unsigned)kRing) {
                                slot[g] = 0u;
                                par[g] ^= 1u;
                            }
                        }
                    }
                    fpar ^= 1u;
                }
            }
            if (!ok && lane) {
                report_stage(&g_ds_status, 1u, 1u << 8);
                mma_commit(smem_u32(&bar_end));
                mbar_wait(smem_u32(&bar_end), 0u);
            }
            __syncwarp();
            stop_sh = 1;
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n" ::: "memory");
        // ---- a tile group
        const unsigned g = tid / kGT, lt = tid % kGT;
        const unsigned r = lt & 127u, hh = lt >> 7;  // row, half
        const unsigned wg = lt >> 5, gbar = 1u + g;
        const unsigned a0 = smem_u32(smraw) + g * kGroupA;
        uint4 *nat = (uint4 *)(smraw + g * kGroupA);  // natural tile (aliases the digits)
        // this warp's lanes, its half's columns
        const unsigned tcol = tmem + 16u * hh + ((32u * (wg & 3u)) << 16);
        unsigned v[64];  // per register: re lo, re hi, im lo, im hi
        unsigned rpar = 0u, dpar = 0u;
        int m14, m24;  // opaque to the compiler, which would make shifts of them
        unsigned one;
        asm volatile("mov.b32 %0, 16384;\n\tmov.b32 %1, 16777216;\n\tmov.b32 %2, 0x64006400;\n"
                     : "=r"(m14), "=r"(m24), "=r"(one));
        // Lane b of a warp holds the amplitude lane of bit b of a tile's index.
        const unsigned wl = tid & 31u;
        int bit_lane = 0;
        {
            idx_t x = insert_zeros((idx_t)1 << (wl < 28u ? wl : 28u), d.ins_pos, d.nins);
            bit_lane = 63 - __clzll(x);
        }
        auto tile_base = [&](int tl) {
            const bool on = (unsigned)tl >> wl & 1u;
            const unsigned lo = on && bit_lane < 32 ? 1u << bit_lane : 0u;
            const unsigned hi = on && bit_lane >= 32 ? 1u << (bit_lane - 32) : 0u;
            const unsigned l = __reduce_or_sync(0xffffffffu, lo);
            const unsigned h = __reduce_or_sync(0xffffffffu, hi);
            return s + (((unsigned long long)h << 32) | l);
        };
        auto row_offset = [&](int f) { return row_off[f][wl] + row_off[f][32 + wg]; };
        auto load_raw = [&](int tl) {
            const uint4 *p0 = tile_base(tl) + row_offset(0);
            lanes_walk(p0, d.in_e, [&](int j, const uint4 *p) {
                const uint4 x = *p;
                v[4 * j] = x.x;
                v[4 * j + 1] = x.y;
                v[4 * j + 2] = x.z;
                v[4 * j + 3] = x.w;
            });
        };
        // the largest of the group's values, to every thread
        auto group_max = [&](unsigned x) {
            x = __reduce_max_sync(0xffffffffu, x);
            if ((tid & 31u) == 0u) red[g][rpar][wg] = x;
            group_sync(gbar, kGT);
            unsigned m = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) m = max(m, red[g][rpar][k]);
            rpar ^= 1u;
            return m;
        };
        auto digits_ready = [&]() {  // this warp's digits are in place
            fence_async_smem();
            __syncwarp();
            if ((tid & 31u) == 0u) mbar_arrive(smem_u32(&bar_a[g]));
        };
        const int tstep = 2 * (int)gridDim.x;
        int tl = (int)(blockIdx.x + g * gridDim.x);
        bool ok = true;
        if (tl < tiles) load_raw(tl);
        for (; tl < tiles && ok; tl += tstep) {
            if (lt == 0u) beat_sh[g] = beat_sh[g] + 1u;
            // the largest component and the smallest amplitude (less 1; zeros are not
            // looked at) of the tile
            unsigned mx = 0, least = 0xffffffffu;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const unsigned a = max(v[4 * j + 1] & 0x7fffffffu, v[4 * j + 3] & 0x7fffffffu);
                mx = max(mx, a);
                least = min(least, a - 1u);
            }
            {
                mx = __reduce_max_sync(0xffffffffu, mx);
                least = __reduce_min_sync(0xffffffffu, least);
                if (wl == 0u) range_sh[g][rpar][wg] = make_uint2(mx, least);
                group_sync(gbar, kGT);
                const uint4 *r4 = (const uint4 *)range_sh[g][rpar];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 x = r4[k];
                    mx = max(mx, max(x.x, x.z));
                    least = min(least, min(x.y, x.w));
                }
                rpar ^= 1u;
            }
            // (a tile of zeros, or of subnormals, stays as it is; components of
            // 2^1018 and more have no room for the digits' constant)
            const bool zero = mx < 0x00100000u, bad = mx >= 0x7fa00000u;
            if (zero || bad) {
                if (bad) {
                    // infinities and NaN spread over the tile as NaN (the CUDA
                    // cores' FP32 pairs would read them as numbers)
                    uint4 *p0 = tile_base(tl) + row_offset(0);
                    lanes_walk(p0, d.in_e, [&](int, uint4 *p) {
                        *p = make_uint4(0u, 0x7ff80000u, 0u, 0x7ff80000u);
                    });
                }
                if (tl + tstep < tiles) load_raw(tl + tstep);
                continue;
            }
            // amplitudes 2^kSkipBits below the largest before the gates: some will be
            // as small after them, so that the tile's blocks would be run in vain
            if ((mx >> 20) > (least >> 20) + kSkipBits && (int)(mx >> 20) >= kRangeLow &&
                (int)(mx >> 20) < kRangeHigh) {
                if (lt == 0u) marks.tile[atomicAdd(&marks.count[0], 1u)] = (unsigned)tl;
                if (tl + tstep < tiles) load_raw(tl + tstep);
                continue;
            }
            // the exponent of the largest component, one more when its
            // mantissa lies within 3 % of the next (the top digit stays below
            // 498 with its carry)
            const int emax = (int)((mx + 0x8000u) >> 20);
            int E = emax - 1071;  // value = V * 2^E
            if (tl + tstep < tiles) {
                // the next tile's 512 lines of 128 bytes on their way to L2
                // while this one's blocks run: two per thread
                const uint4 *p0 = tile_base(tl + tstep) + row_offset(0);
                const unsigned c = r & 7u;  // position in the line: rows' bits 0..2
                for (int b = 0; b < 3; ++b)
                    if (c & (1u << b)) p0 -= 1LL << d.row_lane[b];
                for (int k = 0; k < 3; ++k)
                    if (c & (1u << k)) p0 += d.in_e[k];
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p0));
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p0 + d.in_e[4]));
            }
            unsigned offset = 0u;  // v: integers, value = (V - offset) 2^E
            int top = 0, low = 0;  // range of their high words
            int b = 0;
            // Phase ops from op b on: every amplitude times its table entry, in
            // place.
            auto phase_ops = [&]() {
                while (b < nb && d.op_kind[b] == 1) {
                    const int4 *tab = (const int4 *)(d.bmats + d.op_off[b]);
                    slots_walk(sset[b], r, hh, [&](int j, unsigned slot) {
                        int4 p;
                        asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];\n"
                                     : "=r"(p.x), "=r"(p.y), "=r"(p.z), "=r"(p.w)
                                     : "l"(tab + slot));
                        phase_mul(v, j, offset, p);
                    });
                    offset = 0u;
                    ++b;
                }
                top = low = 0;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    top = max(top, (int)v[2 * j + 1]);
                    low = min(low, (int)v[2 * j + 1]);
                }
            };
            // The integers' digits for dense op b.
            auto split = [&]() {
                const unsigned most = group_max((unsigned)max(top, ~low));
                // V 2^-sh below 0.97 * 2^49 (2^48 for an op_low op)
                int sh = 15 - __clz((int)(most + (most >> 5) + 1u)) + (int)d.op_low[b];
                E += sh;
                unsigned off = PH ? offset : kOffset;
                if (sh < 3) {
                    // a tile that shrank: scaled up
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const unsigned long long V = (join64(v[2 * j], v[2 * j + 1]) - off) << (3 - sh);
                        v[2 * j] = (unsigned)V;
                        v[2 * j + 1] = (unsigned)(V >> 32);
                    }
                    off = 0u;
                    sh = 3;
                }
                // (+ half a unit of the last digit's eighths)
                const unsigned long long bias = (kBias << sh) + ((1ull << sh) >> 4) - off;
                slots_walk(sset[b], r, hh, [&](int j, unsigned slot) {
                    put_digits(a0 + 4u * slot, join64(v[4 * j], v[4 * j + 1]) + bias,
                               join64(v[4 * j + 2], v[4 * j + 3]) + bias, sh, one);
                });
            };
            if (PH && d.op_kind[0] == 1) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const unsigned long long V =
                        biased_from_double(v[2 * j], v[2 * j + 1], emax) - 8ull * kBias;
                    v[2 * j] = (unsigned)V;
                    v[2 * j + 1] = (unsigned)(V >> 32);
                }
                E -= 3;
                phase_ops();
                if (b < nb) split();
            } else {
                // (One rounded FP64 addition of a constant per component gives
                // the biased integers as well, a bit shorter; for half of them
                // that measured 4 % faster, for all of them slower, as that
                // pipe does two operations per cycle and SM.)
                const int etop = emax + (int)d.op_low[0];
                E += (int)d.op_low[0];
                slots_walk(sset[0], r, hh, [&](int j, unsigned slot) {
                    put_digits(a0 + 4u * slot, biased_from_double(v[4 * j], v[4 * j + 1], etop),
                               biased_from_double(v[4 * j + 2], v[4 * j + 3], etop), 3, one);
                });
            }
            while (b < nb) {  // the digits of dense op b are in place
                digits_ready();
                top = low = 0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (ok && !mbar_wait(smem_u32(&bar_d[g][h]), dpar)) ok = false;
                    tc_fence_after();
#pragma unroll
                    for (int c4 = 0; c4 < 4; ++c4) {
                        unsigned L[7][4];
#pragma unroll
                        for (int l = 0; l < 7; ++l)
                            tmem_ld_x4(tcol + (unsigned)h * kHalfCols + (unsigned)l * kLevelCols +
                                           4u * (unsigned)c4,
                                       L[l]);
                        tmem_wait_ld();
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int at = 4 * (2 * c4 + (k >> 1) + 8 * h) + 2 * (k & 1);
                            combine_levels(L[0][k], L[1][k], L[2][k], L[3][k], L[4][k], L[5][k],
                                           L[6][k], m14, m24, v[at], v[at + 1]);
                            top = max(top, (int)v[at + 1]);
                            low = min(low, (int)v[at + 1]);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if ((tid & 31u) == 0u) mbar_arrive(smem_u32(&bar_dfree[h]));
                }
                dpar ^= 1u;
                E += d.op_exp[b] - 4;
                offset = kOffset;
                ++b;
                if (PH && b < nb && d.op_kind[b] == 1) phase_ops();
                if (b < nb) split();
            }
            if (!ok) {
                abort_sh[g] = 1;
                report_stage(&g_ds_status, 2u, 2u << 8);
            }
            {
                // the smallest amplitude (high words; the bits of either part stand
                // for the larger one, within a factor of two)
                unsigned least = 0xffffffffu;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int re = (int)v[4 * j + 1], im = (int)v[4 * j + 3];
                    least = min(least, (unsigned)((re ^ (re >> 31)) | (im ^ (im >> 31))));
                }
                if (least < kLeast && emax >= kRangeLow && emax < kRangeHigh) wide_sh[g] = tl + 1;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j)
                double_from_fixed(v[2 * j], v[2 * j + 1], PH ? offset : kOffset, E);
            // one decision for the whole group (its products are read: the
            // digit buffers are free)
            group_sync(gbar, kGT);
            if (*(volatile int *)&abort_sh[g]) {
                ok = false;
                break;
            }
            if (wide_sh[g] == tl + 1) {
                if (lt == 0u) marks.tile[atomicAdd(&marks.count[0], 1u)] = (unsigned)tl;
                if (tl + tstep < tiles) load_raw(tl + tstep);
                continue;
            }
            if (d.direct_out) {
                // rows in whole 128-byte lines go straight to the state
                uint4 *p0 = tile_base(tl) + row_offset(1);
                lanes_walk(p0, d.out_e, [&](int j, uint4 *p) {
                    *p = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                });
                if (tl + tstep < tiles) load_raw(tl + tstep);
                continue;
            }
            slots_walk(sset[nb], r, hh, [&](int j, unsigned slot) {
                nat[slot] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            });
            group_sync(gbar, kGT);
            if (tl + tstep < tiles) load_raw(tl + tstep);
            {
                uint4 *p = tile_base(tl) + row_offset(0);
                slots_walk(sset[nb + 1], r, hh, [&](int j, unsigned slot) {
                    long long o = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (j >> k & 1) o += d.in_e[k == 3 ? 4 : k];
                    p[o] = nat[slot];
                });
            }
            group_sync(gbar, kGT);  // the natural tile is read before the next digits
        }
        // tells the issuing warp that this group is done
        if (lt == 0u) done_sh[g] = 1;
        group_sync(gbar, kGT);
        __threadfence_block();
        if ((tid & 31u) == 0u) mbar_arrive(smem_u32(&bar_a[g]));
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                     "r"(512u)
                     : "memory");
    }
}

// Diagonal gates alone: every amplitude times its table entry, in FP64.  1024
// amplitudes per CTA and step, four per thread; the table's index is the sum of
// a part by the thread, two by the register and one by the step.  Bound by HBM and
// the FP64 pipe alike (four multiply-adds per amplitude at two per cycle and SM,
// 0.23 ms for 25 lanes; HBM 0.16): 0.26 ms, against 0.44 as a phase op of k_dstage.
struct PhaseLanes {
    int n;
    signed char lane[kMaxPhaseLanes];  // ascending
};
__global__ void __launch_bounds__(256)
k_phase_f64(double2 *__restrict__ s, idx_t chunks, const __grid_constant__ PhaseLanes d,
            const double2 *__restrict__ table) {
    const unsigned tid = threadIdx.x;
    unsigned at = 0, r0 = 0, r1 = 0;
    for (int k = 0; k < d.n; ++k) {
        const int l = d.lane[k];
        if (l < 8) at |= (tid >> l & 1u) << k;
        if (l == 8) r0 = 1u << k;
        if (l == 9) r1 = 1u << k;
    }
    for (idx_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        unsigned slot = at;
        for (int k = 0; k < d.n; ++k)
            if (d.lane[k] >= 10) slot |= (unsigned)(c >> (d.lane[k] - 10) & 1) << k;
        double2 *p = s + (c << 10) + tid;
        double2 x[4], f[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            x[u] = p[256 * u];
            f[u] = __ldg(&table[slot + (u & 1 ? r0 : 0u) + (u & 2 ? r1 : 0u)]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            p[256 * u] = make_double2(x[u].x * f[u].x - x[u].y * f[u].y,
                                      x[u].x * f[u].y + x[u].y * f[u].x);
    }
}

constexpr size_t dstage_smem(int nops) {
    return 2 * (size_t)kGroupA + 2 * (size_t)kRing * kChunk + sizeof(SetSlots) * (size_t)(nops + 2);
}

}  // namespace

void launch_phase_f64(void *state, int n, const int *lanes, int n_lanes, const void *table,
                      cudaStream_t stream) {
    if (n < 10 || n_lanes < 0 || n_lanes > kMaxPhaseLanes)
        fail(2, "phase pass: bad lane counts %d, %d", n, n_lanes);
    PhaseLanes d;
    d.n = n_lanes;
    for (int k = 0; k < n_lanes; ++k) {
        if (lanes[k] < 0 || lanes[k] >= n) fail(2, "phase pass: lane %d outside the state", lanes[k]);
        d.lane[k] = (signed char)lanes[k];
    }
    const idx_t chunks = (idx_t)1 << (n - 10);
    k_phase_f64<<<(unsigned)std::min<idx_t>(chunks, 152 * 8), 256, 0, stream>>>(
        (double2 *)state, chunks, d, (const double2 *)table);
    QG_CUDA(cudaGetLastError());
}

void launch_dstage(void *state, const TcStageDesc &d, const TileMarks &marks, cudaStream_t stream) {
    if (d.m != 12) fail(2, "complex128 tensor stage: tile lanes must be 12 (got %d)", d.m);
    if (d.nblocks < 1 || d.nblocks > kMaxTcBlocks)
        fail(2, "complex128 tensor stage: bad op count %d", d.nblocks);
    if (((uintptr_t)d.bmats & 15u) != 0) fail(2, "complex128 tensor stage: operands misaligned");
    for (int b = 0; b < d.nblocks + 2; ++b) {
        // every slot (an XOR of table entries) stays below the OR of them all
        unsigned any = 0;
        for (unsigned short x : d.sets[b].lo) any |= x;
        for (unsigned short x : d.sets[b].hi) any |= x;
        for (unsigned short x : d.sets[b].q) any |= x;
        if (any >= 4096u) fail(2, "complex128 tensor stage: slot table %d outside the tile", b);
        if (b >= d.nblocks) continue;
        if (d.op_kind[b] > 1) fail(2, "complex128 tensor stage: op %d of unknown kind", b);
        const unsigned need = d.op_kind[b] ? 16u * (any + 1u) : kDigitOpBytes;
        if ((d.op_off[b] & 15u) != 0 || d.op_off[b] + need > d.ops_bytes)
            fail(2, "complex128 tensor stage: op %d operands outside the operand array", b);
    }
    if (d.n < d.m || d.n - d.m > 28) fail(2, "complex128 tensor stage: bad lane count %d", d.n);
    const int tiles = 1 << (d.n - d.m);
    int dev = 0, sms = 0;
    QG_CUDA(cudaGetDevice(&dev));
    QG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const size_t smem = dstage_smem(d.nblocks);
    bool phases = false, dense = false;
    for (int b = 0; b < d.nblocks; ++b) {
        phases = phases || d.op_kind[b] != 0;
        dense = dense || d.op_kind[b] == 0;
    }
    if (!dense) fail(2, "complex128 tensor stage: no dense op");
    auto launch = [&](auto kern) {
        QG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)dstage_smem(kMaxTcBlocks)));
        kern<<<(unsigned)std::min(tiles, sms), kThreads, smem, stream>>>((uint4 *)state, d, tiles,
                                                                         marks);
    };
    phases ? launch(k_dstage<true>) : launch(k_dstage<false>);
    QG_CUDA(cudaGetLastError());
}

__global__ void k_raise_dstage(unsigned bits) { report_stage(&g_ds_status, bits, bits << 8); }

void dstage_status_host(unsigned *word) {
    const StageStatus s = {0u, word};
    QG_CUDA(cudaMemcpyToSymbol(g_ds_status, &s, sizeof(s)));
}

void dstage_raise(unsigned bits, cudaStream_t stream) {
    k_raise_dstage<<<1, 1, 0, stream>>>(bits);
    QG_CUDA(cudaGetLastError());
}

int dstage_status(bool reset) {
    unsigned v = 0;
    QG_CUDA(cudaMemcpyFromSymbol(&v, g_ds_status, sizeof(v)));
    if (reset && v) {
        const unsigned z = 0;
        QG_CUDA(cudaMemcpyToSymbol(g_ds_status, &z, sizeof(z)));
    }
    return (int)v;
}

}  // namespace qg
