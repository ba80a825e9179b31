// Kernels of the adjoint-differentiation engine (sm_103a).
//
// A batch of B parameter vectors of one circuit shares one stage program;
// each CTA handles one tile of one batch element (grid = tiles x B) and reads
// that element's gate matrices from a per-element table.  The backward stage
// keeps the tiles of both psi and lambda = U^dagger ... H psi in registers,
// and for every parametrised rotation exp(-i c theta G) it first accumulates
// Im<lambda|P1 G|psi> (P1: its controls set) and then un-applies the gate to
// both states -- the gradient is 2c times that sum.  One HBM read and write of
// psi and lambda per stage, however many gates it holds.
//
// The reference has no differentiation path; its nearest composition is
// finite differences or parameter-shift over repeated runs
// (qgate/simulator/simulator.py:57-83 per evaluation).
#include "qg_regstage.cuh"

namespace qg {

namespace {

using namespace rs;

template <class C> __device__ __forceinline__ auto im_conj_mul(C l, C p) {  // Im(conj(l) p)
    return l.x * p.y - l.y * p.x;
}
template <class C> __device__ __forceinline__ auto re_conj_mul(C l, C p) {  // Re(conj(l) p)
    return l.x * p.x + l.y * p.y;
}

// Im<lam|P1 G|psi> over this thread's register pairs on register bit I.
template <int I, int NR, class C, class R>
__device__ __forceinline__ void reg_grad(const C (&a)[NR], const C (&l)[NR], unsigned jmask,
                                         int axis, R &out) {
    R acc = 0;
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        if (j & (1 << I)) continue;
        if ((j & jmask) != jmask) continue;
        const C p0 = a[j], p1 = a[j | (1 << I)], l0 = l[j], l1 = l[j | (1 << I)];
        if (axis == 1)
            acc += im_conj_mul(l0, p1) + im_conj_mul(l1, p0);
        else if (axis == 2)
            acc += re_conj_mul(l1, p0) - re_conj_mul(l0, p1);
        else
            acc += im_conj_mul(l0, p0) - im_conj_mul(l1, p1);
    }
    out = acc;
}

// Shared-memory bytes of n register-set slot tables, rounded to 16.
__host__ __device__ constexpr unsigned adj_sets_bytes(int nsets) {
    return ((unsigned)nsets * (unsigned)sizeof(SetSlots) + 15u) & ~15u;
}

template <class R> __device__ __forceinline__ R warp_sum(R v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Global offset of register j: the sum of e[k] over the set bits k of j.
template <int RL> __device__ __forceinline__ idx_t reg_offset(const idx_t (&e)[RL], int j) {
    idx_t o = 0;
#pragma unroll
    for (int k = 0; k < RL; ++k)
        if (j & (1 << k)) o += e[k];
    return o;
}

// CTAs per SM the registers leave room for.  complex64 backward stages: five (48
// registers without spills) against four 20.4 and 20.7 ms for the gradient below,
// 14.6 and 15.1 ms without checkpoints; six spill (21.2 and 15.1 ms).
template <class R, int RL, int MODE>
constexpr int kAdjBlocks = MODE == 1 && RL == 3 && sizeof(R) == 4 ? 5 : 0;

// Backward stages read psi and lambda and write lambda (psi too where no
// checkpoint follows): HBM sets the floor, 60 us for 16 vectors of 20 qubits.  A
// stage whose register set holds none of the lowest lanes runs from global loads
// to global stores in registers, without shared memory or its barriers; with
// several sets the first and the last do so.  Psi is carried only as far as the
// last gradient where nothing reads it after, and not read without one.  20 qubits,
// 6 layers, batch 16, a checkpoint every 3 gates: a stage of diagonal rotations
// 90 us, of RY 97, of CX (lambda alone: 40 us of HBM) 61; 96 to 111 before, when
// every stage went through shared memory with both states.  What is left is issue
// (runtime control masks on every register).
template <class R, int RL, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? 256 : 512, kAdjBlocks<R, RL, MODE>)
k_adj_stage(const typename CT<R>::type *psi_src, typename CT<R>::type *psi_dst,
            typename CT<R>::type *lam_all, int store_lam, const __grid_constant__ AdjStageDesc d,
            const R *__restrict__ mats_all, R *__restrict__ gpart, int slot_stride) {
    typedef typename CT<R>::type C;
    constexpr int NR = 1 << RL;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int m = d.m, n = d.n;
    const unsigned tid = threadIdx.x, T = blockDim.x;
    const int b = blockIdx.y;
    const idx_t tiles = (idx_t)gridDim.x;
    const C *psi = psi_src + ((idx_t)b << n);
    C *lam = MODE == 1 ? lam_all + ((idx_t)b << n) : nullptr;

    const unsigned tile = adj_in_registers(d) ? 0u : 1u << m;
    C *sp = (C *)smraw;
    C *sl = sp + (MODE == 1 ? tile : 0u);
    AdjOp *sops = (AdjOp *)(sp + (MODE == 1 ? 2u : 1u) * tile);
    SetSlots *sset = (SetSlots *)(sops + d.nops);
    R *smat = (R *)((unsigned char *)sset + adj_sets_bytes(d.nsets));
    R *sgrad = smat + 8 * d.nmats;

    // psi goes nowhere when a checkpoint replaces it next, lambda when no
    // rotation is left before it
    const bool keep_psi = MODE == 0 || psi_dst != nullptr, keep_lam = MODE == 1 && store_lam;
    const bool use_psi = keep_psi || d.last_grad >= 0;
    const int t = m - RL;
    const idx_t base = insert_zeros((idx_t)blockIdx.x, d.ins_pos, d.nins);
    auto thread_offset = [&](int f) {
        idx_t o = base;
        for (int k = 0; k < t; ++k)
            if (tid >> k & 1u) o |= 1LL << d.io_lane[f][k];
        return o;
    };
    auto register_lanes = [&](int f, idx_t (&e)[RL]) {
#pragma unroll
        for (int k = 0; k < RL; ++k) e[k] = 1LL << d.io_lane[f][t + k];
    };
    const unsigned pt = Swz<R>::f(tid);
    C a[NR], l[NR];
    {
        const idx_t g0 = thread_offset(0);
        idx_t e[RL];
        register_lanes(0, e);
        if (d.direct_in) {
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                const idx_t g = g0 + reg_offset<RL>(e, j);
                if (MODE == 0 && !psi_src)
                    a[j] = cmk<C>(g == 0 ? 1. : 0., 0.);  // |0...0>
                else if (use_psi)
                    a[j] = psi[g];
                if (MODE == 1) l[j] = lam[g];
            }
        } else {
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const unsigned slot = pt ^ Swz<R>::f((unsigned)i << t);
                const idx_t g = g0 + reg_offset<RL>(e, i);
                if (MODE == 0 && !psi_src)
                    sp[slot] = cmk<C>(g == 0 ? 1. : 0., 0.);  // |0...0>
                else if (use_psi)
                    cp_async_elem(&sp[slot], &psi[g]);
                if (MODE == 1) cp_async_elem(&sl[slot], &lam[g]);
            }
        }
    }
    {
        const int4 *src = (const int4 *)d.ops;
        int4 *dst = (int4 *)sops;
        for (int i = tid; i < d.nops; i += T) dst[i] = src[i];
        copy_sets(sset, d.sets, d.nsets, tid, T);
        const R *mats = mats_all + (size_t)b * d.nmats * 8;
        for (int i = tid; i < 8 * d.nmats; i += T) smat[i] = mats[i];
        if (MODE == 1)
            for (int i = tid; i < d.ngrads; i += T) sgrad[i] = 0;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();

    unsigned e0 = 0, P0 = 0;
    unsigned q[RL];
#pragma unroll
    for (int k = 0; k < RL; ++k) q[k] = 0;
    const unsigned lane = tid & 31u;

    for (int oi = 0; oi < d.nops; ++oi) {
        const AdjOp o = sops[oi];
        // whether the op has to change psi, lambda
        const bool on_psi = keep_psi || oi < d.last_grad;
        const bool on_lam = MODE == 1 && (keep_lam || oi < d.last_grad);
        if (o.kind == kOpTranspose) {
            if (oi > 0) {
                __syncthreads();
#pragma unroll
                for (int j = 0; j < NR; ++j) {
                    unsigned sl_ = reg_slot<RL>(P0, q, j);
                    if (on_psi) sp[sl_] = a[j];
                    if (on_lam) sl[sl_] = l[j];
                }
                __syncthreads();
            }
            const SetSlots &ss = sset[o.reg];
            P0 = (unsigned)ss.lo[tid & 31u] ^ (unsigned)ss.hi[tid >> 5];
            e0 = Swz<R>::f(P0);
#pragma unroll
            for (int k = 0; k < RL; ++k) q[k] = ss.q[k];
            if (oi == 0 && d.direct_in) continue;
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                unsigned sl_ = reg_slot<RL>(P0, q, j);
                if (on_psi) a[j] = sp[sl_];
                if (on_lam) l[j] = sl[sl_];
            }
            continue;
        }
        const bool act = (e0 & o.tmask) == o.tmask;
        if (MODE == 1 && o.gaxis) {
            R v = 0;
            if (act) {
                if (o.kind == kOpDiagThread) {
                    R acc = 0;
#pragma unroll
                    for (int j = 0; j < NR; ++j)
                        if ((j & o.jmask) == o.jmask) acc += im_conj_mul(l[j], a[j]);
                    v = (e0 & o.tbit) ? -acc : acc;
                } else {
                    QG_REG_DISPATCH(reg_grad, o.reg, a, l, (unsigned)o.jmask, (int)o.gaxis, v);
                }
            }
            v = warp_sum(v);
            if (lane == 0) atomicAdd(&sgrad[o.gslot], v);
        }
        if (!act) continue;
        const R *mm_ = smat + 8 * o.mat;
        if (o.kind == kOpGate) {
            MatR<R> mm;
            mm.m00 = cmk<C>(mm_[0], mm_[1]);
            mm.m01 = cmk<C>(mm_[2], mm_[3]);
            mm.m10 = cmk<C>(mm_[4], mm_[5]);
            mm.m11 = cmk<C>(mm_[6], mm_[7]);
            if (on_psi) QG_REG_DISPATCH(reg_gate, o.reg, a, mm, (unsigned)o.jmask);
            if (on_lam) QG_REG_DISPATCH(reg_gate, o.reg, l, mm, (unsigned)o.jmask);
        } else if (o.kind == kOpSwapX) {
            if (on_psi) QG_REG_DISPATCH(reg_swap, o.reg, a, (unsigned)o.jmask);
            if (on_lam) QG_REG_DISPATCH(reg_swap, o.reg, l, (unsigned)o.jmask);
        } else if (o.kind == kOpDiagReg) {
            C d0 = cmk<C>(mm_[0], mm_[1]), d1 = cmk<C>(mm_[6], mm_[7]);
            if (on_psi) QG_REG_DISPATCH(reg_diag, o.reg, a, d0, d1, (unsigned)o.jmask);
            if (on_lam) QG_REG_DISPATCH(reg_diag, o.reg, l, d0, d1, (unsigned)o.jmask);
        } else {  // kOpDiagThread
            C ph = (e0 & o.tbit) ? cmk<C>(mm_[6], mm_[7]) : cmk<C>(mm_[0], mm_[1]);
#pragma unroll
            for (int j = 0; j < NR; ++j)
                if ((j & o.jmask) == o.jmask) {
                    if (on_psi) a[j] = cmul(ph, a[j]);
                    if (on_lam) l[j] = cmul(ph, l[j]);
                }
        }
    }

    __syncthreads();
    if (keep_psi || keep_lam) {
        const idx_t g0 = thread_offset(1);
        idx_t e[RL];
        register_lanes(1, e);
        C *out = psi_dst + ((idx_t)b << n);
        if (d.direct_out) {
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                const idx_t g = g0 + reg_offset<RL>(e, j);
                if (keep_psi) out[g] = a[j];
                if (keep_lam) lam[g] = l[j];
            }
        } else {
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                unsigned sl_ = reg_slot<RL>(P0, q, j);
                if (keep_psi) sp[sl_] = a[j];
                if (keep_lam) sl[sl_] = l[j];
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const unsigned slot = pt ^ Swz<R>::f((unsigned)i << t);
                const idx_t g = g0 + reg_offset<RL>(e, i);
                if (keep_psi) out[g] = sp[slot];
                if (keep_lam) lam[g] = sl[slot];
            }
        }
    }
    if (MODE == 1)
        for (int i = tid; i < d.ngrads; i += T)
            gpart[((idx_t)b * slot_stride + i) * tiles + blockIdx.x] = sgrad[i];
}

// sums[b * nslots + s] = sum over tiles of slot s's partials, FP64.
template <class R>
__global__ void k_adj_grad_reduce(const R *__restrict__ partials, int slot_stride, idx_t tiles,
                                  double *__restrict__ sums, int nslots) {
    const int s = blockIdx.x, b = blockIdx.y;
    const R *p = partials + ((idx_t)b * slot_stride + s) * tiles;
    double acc = 0.;
    for (idx_t i = threadIdx.x; i < tiles; i += blockDim.x) acc += (double)p[i];
    __shared__ double ws[32];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += ws[w];
        sums[(idx_t)b * nslots + s] = v;
    }
}

struct PauliTerms {
    int n;
    PauliTerm t[kMaxPauliTerms];
};

// lam[i] = sum_t coef_t i^ny_t (-1)^popcount((i ^ x_t) & z_t) psi[i ^ x_t]
// and the block partials of Re<psi|lam> (FP64 per block).  Bound by issue: 39
// terms of a 20-qubit Ising chain on 2^24 amplitudes, whose bytes take 0.04 ms.
// A thread holds four amplitudes 256 apart, so that a term's parity is formed
// once and flipped by two bits of its z mask; one amplitude per thread with its
// own parity and the amplitude itself loaded again for every Z term took 1.28 ms,
// this 0.49 ms.
__device__ __forceinline__ float flip_sign(float c, unsigned odd) {
    return __uint_as_float(__float_as_uint(c) ^ (odd << 31));
}
__device__ __forceinline__ double flip_sign(double c, unsigned odd) {
    return __hiloint2double((int)((unsigned)__double2hiint(c) ^ (odd << 31)), __double2loint(c));
}
template <class R>
__global__ void __launch_bounds__(256)
k_pauli_sum_apply(const typename CT<R>::type *__restrict__ psi_all,
                  typename CT<R>::type *__restrict__ lam_all, int n,
                  const __grid_constant__ PauliTerms terms, double *__restrict__ e_partials) {
    typedef typename CT<R>::type C;
    constexpr int U = 4;
    const int b = blockIdx.y;
    const idx_t N = (idx_t)1 << n;
    const C *psi = psi_all + (idx_t)b * N;
    C *lam = lam_all + (idx_t)b * N;
    double acc = 0.;
    const int held = N < 256 * U ? (int)((N + 255) >> 8) : U;  // amplitudes of a thread
    const idx_t stride = (idx_t)gridDim.x * (256 * U);
    for (idx_t i = (idx_t)blockIdx.x * (256 * U) + threadIdx.x; i < N; i += stride) {
        C p[U];
        R re[U], im[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            re[u] = im[u] = 0;
            if (u < held) p[u] = psi[i + 256 * u];
        }
        for (int k = 0; k < terms.n; ++k) {
            const PauliTerm &pt = terms.t[k];
            const unsigned long long x = (unsigned long long)pt.x, z = (unsigned long long)pt.z;
            const unsigned long long zs = ((unsigned long long)i ^ x) & z;
            const unsigned odd = (unsigned)__popc((unsigned)zs ^ (unsigned)(zs >> 32)) & 1u;
            const int ny = __popcll(x & z) & 3;
            const R coef = (R)pt.coef;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (u >= held) continue;
                const unsigned flip = (u & 1 ? (unsigned)(z >> 8) : 0u) ^
                                      (u & 2 ? (unsigned)(z >> 9) : 0u);
                const R c = flip_sign(coef, (odd ^ flip) & 1u);
                const C v = x ? psi[(i + 256 * u) ^ (idx_t)x] : p[u];
                // multiply v by c * i^ny
                const R vr = v.x * c, vi = v.y * c;
                if (ny == 0) {
                    re[u] += vr;
                    im[u] += vi;
                } else if (ny == 1) {
                    re[u] -= vi;
                    im[u] += vr;
                } else if (ny == 2) {
                    re[u] -= vr;
                    im[u] -= vi;
                } else {
                    re[u] += vi;
                    im[u] -= vr;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u >= held) continue;
            C out;
            out.x = re[u];
            out.y = im[u];
            lam[i + 256 * u] = out;
            acc += (double)(p[u].x * re[u] + p[u].y * im[u]);
        }
    }
    acc = warp_sum(acc);
    __shared__ double ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.;
        for (int w = 0; w < 8; ++w) v += ws[w];
        e_partials[(idx_t)b * gridDim.x + blockIdx.x] = v;
    }
}

__global__ void k_sum_rows(const double *__restrict__ partials, int cols, double *out) {
    double acc = 0.;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) acc += partials[(idx_t)blockIdx.x * cols + i];
    acc = warp_sum(acc);
    __shared__ double ws[32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += ws[w];
        out[blockIdx.x] = v;
    }
}

constexpr int kPauliBlocks = 152 * 2;

template <class R, int MODE>
void adj_dispatch(const void *psi_src, void *psi_dst, void *lam, bool store_lam,
                  const AdjStageDesc &d, const void *mats, void *gpart, int slot_stride, int batch,
                  cudaStream_t stream) {
    typedef typename CT<R>::type C;
    const size_t tile = adj_in_registers(d) ? 0 : (sizeof(C) << d.m) * (MODE == 1 ? 2 : 1);
    size_t smem = tile + (size_t)d.nops * sizeof(AdjOp) + adj_sets_bytes(d.nsets) +
                  sizeof(R) * (8 * (size_t)d.nmats + (size_t)d.ngrads);
    idx_t tiles = (idx_t)1 << (d.n - d.m);
    int threads = 1 << (d.m - d.rl);
    dim3 grid((unsigned)tiles, (unsigned)batch);
    auto launch = [&](auto kern) {
        QG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, threads, smem, stream>>>((const C *)psi_src, (C *)psi_dst, (C *)lam,
                                              store_lam ? 1 : 0, d, (const R *)mats, (R *)gpart,
                                              slot_stride);
    };
    switch (d.rl) {
    case 3: launch(k_adj_stage<R, 3, MODE>); break;
    case 4: launch(k_adj_stage<R, 4, MODE>); break;
    case 5:
        // forward stages of complex64 only (the backward holds psi and
        // lambda: 2 x 32 amplitudes per thread would not fit)
        if constexpr (MODE == 0 && sizeof(R) == 4)
            launch(k_adj_stage<R, 5, MODE>);
        else
            fail(2, "adjoint stage: 5 register lanes only for complex64 forward stages");
        break;
    default: fail(2, "adjoint stage: unsupported register lanes %d", d.rl);
    }
    QG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_adj_stage(int prec, int mode, const void *psi_src, void *psi_dst, void *lam,
                      bool store_lam, const AdjStageDesc &d, const void *mats,
                      void *grad_partials, int slot_stride, int batch, cudaStream_t stream) {
    auto run = [&](auto dispatch) {
        dispatch(psi_src, psi_dst, lam, store_lam, d, mats, grad_partials, slot_stride, batch,
                 stream);
    };
    if (prec == kFP32) {
        if (mode == 0)
            run(adj_dispatch<float, 0>);
        else
            run(adj_dispatch<float, 1>);
    } else {
        if (mode == 0)
            run(adj_dispatch<double, 0>);
        else
            run(adj_dispatch<double, 1>);
    }
}

void launch_adj_grad_reduce(int prec, const void *partials, int batch, int slots, int slot_stride,
                            idx_t tiles, double *sums, int nslots, cudaStream_t stream) {
    if (slots == 0) return;
    dim3 grid((unsigned)slots, (unsigned)batch);
    if (prec == kFP32)
        k_adj_grad_reduce<float><<<grid, 256, 0, stream>>>((const float *)partials, slot_stride,
                                                           tiles, sums, nslots);
    else
        k_adj_grad_reduce<double><<<grid, 256, 0, stream>>>((const double *)partials, slot_stride,
                                                            tiles, sums, nslots);
    QG_CUDA(cudaGetLastError());
}

int pauli_sum_blocks() { return kPauliBlocks; }

void launch_pauli_sum_apply(int prec, const void *psi, void *lam, int n, int batch,
                            const PauliTerm *terms, int nterms, double *e_partials,
                            int blocks_per_batch, cudaStream_t stream) {
    if (nterms > kMaxPauliTerms) fail(1, "at most %d Pauli terms", kMaxPauliTerms);
    PauliTerms pt;
    pt.n = nterms;
    for (int i = 0; i < nterms; ++i) pt.t[i] = terms[i];
    dim3 grid((unsigned)blocks_per_batch, (unsigned)batch);
    if (prec == kFP32)
        k_pauli_sum_apply<float><<<grid, 256, 0, stream>>>((const float2 *)psi, (float2 *)lam, n, pt,
                                                           e_partials);
    else
        k_pauli_sum_apply<double><<<grid, 256, 0, stream>>>((const double2 *)psi, (double2 *)lam, n,
                                                            pt, e_partials);
    QG_CUDA(cudaGetLastError());
}

void launch_sum_rows(const double *partials, int rows, int cols, double *out, cudaStream_t stream) {
    k_sum_rows<<<rows, 256, 0, stream>>>(partials, cols, out);
    QG_CUDA(cudaGetLastError());
}

}  // namespace qg
