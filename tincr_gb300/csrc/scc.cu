// Batched SCC ground states (restricted closed shell, long-range corrected or not), one system per
// thread-block cluster.
//
// Follows tincr's SCC routine (src/scc/scc_routine.rs:121-290) together with the inputs it builds
// first: overlap S and H0 from the Slater-Koster splines (src/scc/h0_and_s.rs:92-182), the Gaussian
// gamma matrices (src/scc/gamma_approximation.rs:75-124, :175-193), the neutral-atom reference density
// (src/scc/helpers.rs:218-229), the long-range exchange Hamiltonian (src/scc/helpers.rs:111-155), the
// Loewdin orthogonalisation X = S^-1/2 (scc_routine.rs:172-174) and the repulsive energy.
// Convergence: the largest element of the commutator X^T (F P S - S P F) X below tol, with DIIS on the
// Fock matrix (up to 8 iterates).  tincr mixes Mulliken charges with Broyden's method and stops at an
// rms charge change of 1e-5: the same stationary density, reached here to a tighter test.
//
// Layout.  A persistent grid of clusters of 1 to 16 CTAs (two CTAs per SM) takes systems from a counter,
// largest first.  A cluster keeps its system's matrices in a private slot of global memory (a few MB, L2-resident) and
// runs every step itself; its CTAs share out the tiles, rows, roots and elements of a step and meet at
// the cluster barrier, small vectors and sums going straight into each other's shared memory:
//  * the FP64 products of the iterations as exact digit products on warp MMAs (sc_prod); those of small
//    systems, of the set-up and of the FP32 phase on tiles of 16 x 16 outputs, one per thread (FP64), or
//    32 x 32, 2 x 2 per thread (FP32).  GB300 issues 2 FP64 FMAs per SM and clock, 1/64 of its FP32 rate;
//  * the density of an iteration by purification (sc_purify), the eigenpairs of S and of the last Fock
//    matrix (and of one without a gap) by a tridiagonal eigensolver;
//  * eigenpairs: Householder tridiagonalisation, Sturm-count multisection (the lanes that the roots
//    leave idle take more points per root), inverse iteration with one thread per root (LU with partial
//    pivoting), Loewdin's orthogonalisation to first order (Gram-Schmidt inside clusters of close roots
//    where that does not do), and the back-transformation by the stored reflections;
//  * the Fock build, Mulliken charges, DIIS and the energy as element loops and reductions.
// CTAs per system: sc_ctas_per_system.  Kernel time (ms, LC, to 1e-10) with one CTA per system, FP64 tiles and
// the eigensolver in every iteration / with clusters / with digit products and purification too:
//     one decacene (192 orbitals)  705 / 123 / 44       128 acene dimers (up to 186)  750 / 417 / 176
//     16 acene dimers              690 / 160 / 54       64 acenes (up to 102)         145 /  74 /  37
//     40 acene dimers              719 / 233 / 79       400 acene dimers             1100 / 1081 / 512
// SC_FILL 2, 4 and 8: 40 dimers 109, 79, 123; 128 dimers 237, 176, 207; 200 dimers 438, 266, 261.  Below
// SC_DIGITS the operand splits and barriers cost more than the FP64 tiles: 66 orbitals on 16 CTAs 10.2 ms
// on tiles, 13.0 on digits.  What bounds it: the latency of the digit products' loads and barriers at
// 16 CTAs per system, the tensor and integer pipes (digit splits) of full batches.
// With TINCR_SCC_FP32_START the iterations run in FP32 until the commutator is below 1e-5 (at most
// SC_FP32_MAX of them), then continue in FP64 from that density with the DIIS history carried over: the
// stationary point, the convergence test and the final orbitals are FP64 either way.  It pays where FP64
// products run on tiles; on digits it costs (529 acene dimers 766 -> 820 ms).
// Every loop is bounded (max_iter, 80 multisection steps, 3 inverse iterations); CTAs wait for each
// other only at cluster barriers, which every thread of a cluster reaches the same number of times
// (decisions come from values that every CTA forms from the same numbers in the same order).
// Non-finite values end the system's iterations and are reported.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include <cooperative_groups.h>

#include "common.cuh"
#include "fixed8.cuh"
#include "sk_math.cuh"
#include "tda.cuh"

namespace cg = cooperative_groups;

namespace tincr {

namespace {

constexpr int SC_T = 256, SC_W = SC_T / 32;
constexpr int SC_NMAX = 256;           // orbitals (and atoms) per system
constexpr int SC_DIIS = 8;             // DIIS history
constexpr int SC_FP32_MAX = 20;        // FP32 iterations at most before the FP64 phase
constexpr double SC_FP32_SWITCH = 1e-5;
constexpr double SC_PROXIMITY = 30.0;  // bohr: Slater-Koster pairs farther apart are zero (tincr's PROXIMITY_CUTOFF)
constexpr int SC_SLOTS_PER_SM = 2;
constexpr int SC_KS = 32;              // k depth of a GEMM slice
constexpr int SC_DIGITS = 20000;       // n^3 per CTA from which the iterations' FP64 products run on digits
constexpr int SC_CMAX = 16;            // CTAs per cluster
constexpr double SC_FILL = 4.0;        // CTAs per SM that a batch of large systems is spread over (twice what runs at once)
constexpr double SC_SMALL = 96.0;      // orbitals below which systems count as small (sc_ctas_per_system)

struct ScArgs {
    int n_sys;
    const tincr_scc_system *sys;
    const int *order;                  // systems in the order they are taken
    const int *kind;
    const double *xyz;
    const double *p_start;             // packed n x n blocks or null
    const double *s_in, *h0_in, *gam_in, *glr_in;   // caller-supplied inputs or null
    // parameter tables
    int n_kinds, n_knots, sk_extrapolate;
    const int *kind_z, *kind_norb, *kind_l, *kind_m;
    const double *kind_occ, *kind_energy, *sigma, *knots, *coef;
    int rep_ntmax;
    const int *rep_nt;
    const double *rep_knots, *rep_coef, *rep_dmax;
    int lc;
    double r_lr, tol, level_shift;
    int max_iter, fp32_start;
    // outputs (null: not wanted)
    double *orbe, *orbs, *p, *dq, *energy, *s_out, *h0_out, *hcx, *residual;
    int *iterations, *converged, *status;
    // slots
    unsigned char *ws;
    long long slot_bytes, nn_max, at2_max, npad;
    int csize;                         // CTAs per cluster (and system)
    int *next;
};

// shared memory of one CTA; arrays that every CTA of a cluster needs are held in each of them
struct ScShared {
    alignas(16) double gemm[2 * SC_KS * 17];            // GEMM tiles (FP64 32 x 17, FP32 32 x 33 each); dot partials
    double d[SC_NMAX], e[SC_NMAX], beta[SC_NMAX], esq[SC_NMAX], vu[SC_NMAX], cur[SC_NMAX];
    double vp[2][SC_NMAX], rb[2][SC_NMAX];               // written by the other CTAs, alternating
    double xch[2][SC_CMAX][SC_DIIS];                     // sums of every CTA, alternating
    double w[SC_NMAX];                                   // eigenvalues
    double qao[SC_NMAX], dq[SC_NMAX], esp[SC_NMAX];
    double red[SC_W * SC_DIIS + SC_DIIS + 8];
    double B[SC_DIIS][SC_DIIS];
    double coef[SC_DIIS + 1];
    double lin[(SC_DIIS + 1) * (SC_DIIS + 2)];
    int kind[SC_NMAX], ao_off[SC_NMAX + 1];
    short ao_atom[SC_NMAX];
    int sys_id;
    int rank, csize, par;   // CTA of the cluster, CTAs, parity of the next exchange
};

// The CTAs of a cluster work on one system.  SC_FOR: an element loop over all their threads;
// sc_bar: what they wrote to global (and to each other's shared) memory is visible after it.
#define SC_FOR(t, count) \
    for (long long t = (long long)sm.rank * SC_T + threadIdx.x; t < (count); t += (long long)sm.csize * SC_T)

__device__ __forceinline__ void sc_bar(const ScShared &sm) {
    if (sm.csize > 1) cg::this_cluster().sync();
    else __syncthreads();
}

// the same variable in CTA r of the cluster
template <class V>
__device__ __forceinline__ V *sc_at(V *x, int r) { return cg::this_cluster().map_shared_rank(x, r); }

// ---------------------------------------------------------------------------------------------
// Reductions (every thread of every CTA receives the result)
// ---------------------------------------------------------------------------------------------

// m sums (m <= SC_DIIS) of the CTA into sm.red[SC_W * SC_DIIS + r], then over the cluster in CTA order
__device__ void sc_sums(double *v, int m, ScShared &sm) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    for (int r = 0; r < m; ++r) {
        double x = v[r];
        for (int off = 16; off; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if (lane == 0) sm.red[warp * SC_DIIS + r] = x;
    }
    __syncthreads();
    const int par = sm.par;
    if (threadIdx.x < m) {
        double s = 0.0;
        for (int w = 0; w < SC_W; ++w) s += sm.red[w * SC_DIIS + threadIdx.x];
        sm.red[SC_W * SC_DIIS + threadIdx.x] = s;
        if (sm.csize > 1)
            for (int c = 0; c < sm.csize; ++c) *sc_at(&sm.xch[par][sm.rank][threadIdx.x], c) = s;
    }
    if (sm.csize > 1) {
        sc_bar(sm);   // a CTA writes this parity again only after the next exchange's barrier
        if (threadIdx.x < m) {
            double s = 0.0;
            for (int c = 0; c < sm.csize; ++c) s += sm.xch[par][c][threadIdx.x];
            sm.red[SC_W * SC_DIIS + threadIdx.x] = s;
        }
        if (threadIdx.x == 0) sm.par = par ^ 1;
    }
    __syncthreads();
}

__device__ double sc_sum(double v, ScShared &sm) {
    sc_sums(&v, 1, sm);
    return sm.red[SC_W * SC_DIIS];
}

// maximum over the CTA
__device__ double sc_max_cta(double v, ScShared &sm) {
    for (int off = 16; off; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sm.red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = sm.red[0];
    for (int w = 1; w < SC_W; ++w) s = fmax(s, sm.red[w]);
    __syncthreads();
    return s;
}

// maximum over the cluster
__device__ double sc_max(double v, ScShared &sm) {
    double s = sc_max_cta(v, sm);
    if (sm.csize > 1) {
        const int par = sm.par;
        if (threadIdx.x < sm.csize) *sc_at(&sm.xch[par][sm.rank][0], (int)threadIdx.x) = s;
        sc_bar(sm);
        for (int c = 0; c < sm.csize; ++c) s = fmax(s, sm.xch[par][c][0]);
        __syncthreads();
        if (threadIdx.x == 0) sm.par = par ^ 1;
        __syncthreads();
    }
    return s;
}

// ---------------------------------------------------------------------------------------------
// GEMM of the cluster: C = alpha op(A) op(B) + beta C, row-major, op(A) M x K, op(B) K x N (beta = 0: C
// not read); the tiles are dealt to the CTAs.
// Tiles of TL = 16 R outputs square; thread (ty, tx) computes rows R ty + i, columns R tx + j.
// ---------------------------------------------------------------------------------------------

template <class T, int R>
__device__ void sc_gemm(int M, int N, int K, T alpha, const T *A, int lda, bool ta, const T *B, int ldb, bool tb,
                        T beta, T *C, int ldc, ScShared &sm, bool sym) {
    constexpr int TL = 16 * R, PE = TL * SC_KS / SC_T;
    T(*As)[TL + 1] = reinterpret_cast<T(*)[TL + 1]>(sm.gemm);
    T(*Bs)[TL + 1] = reinterpret_cast<T(*)[TL + 1]>(reinterpret_cast<T *>(sm.gemm) + SC_KS * (TL + 1));
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int tm = (M + TL - 1) / TL, tn = (N + TL - 1) / TL;
    // symmetric result: the tiles on and below the diagonal, row by row
    const int count = sym ? tm * (tm + 1) / 2 : tm * tn;
    for (int t = sm.rank; t < count; t += sm.csize) {
        int ti = t / tn, tj = t % tn;
        if (sym) {
            ti = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
            while (ti * (ti + 1) / 2 > t) --ti;
            while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
            tj = t - ti * (ti + 1) / 2;
        }
        const int m0 = ti * TL, n0 = tj * TL;
        T acc[R][R];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < R; ++j) acc[i][j] = T(0);
        T ra[PE], rb[PE];
        auto load = [&](int k0) {
#pragma unroll
            for (int q = 0; q < PE; ++q) {
                const int e = tid + q * SC_T;   // 0 .. SC_KS TL - 1
                const int m = m0 + (ta ? e % TL : e / SC_KS), ka = k0 + (ta ? e / TL : e % SC_KS);
                ra[q] = (m < M && ka < K) ? (ta ? A[(long long)ka * lda + m] : A[(long long)m * lda + ka]) : T(0);
                const int n = n0 + (tb ? e / SC_KS : e % TL), kb = k0 + (tb ? e % SC_KS : e / TL);
                rb[q] = (n < N && kb < K) ? (tb ? B[(long long)n * ldb + kb] : B[(long long)kb * ldb + n]) : T(0);
            }
        };
        load(0);
        for (int k0 = 0; k0 < K; k0 += SC_KS) {
            __syncthreads();
#pragma unroll
            for (int q = 0; q < PE; ++q) {
                const int e = tid + q * SC_T;
                As[ta ? e / TL : e % SC_KS][ta ? e % TL : e / SC_KS] = ra[q];
                Bs[tb ? e % SC_KS : e / TL][tb ? e / SC_KS : e % TL] = rb[q];
            }
            __syncthreads();
            if (k0 + SC_KS < K) load(k0 + SC_KS);
            auto step = [&](int kk) {
                T a[R], b[R];
#pragma unroll
                for (int i = 0; i < R; ++i) a[i] = As[kk][R * ty + i];
#pragma unroll
                for (int j = 0; j < R; ++j) b[j] = Bs[kk][R * tx + j];
#pragma unroll
                for (int i = 0; i < R; ++i)
#pragma unroll
                    for (int j = 0; j < R; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            };
            if (K - k0 >= SC_KS) {
#pragma unroll
                for (int kk = 0; kk < SC_KS; ++kk) step(kk);
            } else {
                for (int kk = 0; kk < K - k0; ++kk) step(kk);
            }
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const int m = m0 + R * ty + i, n = n0 + R * tx + j;
                if (m < M && n < N && !(sym && n > m)) {
                    T *c = C + (long long)m * ldc + n;
                    const T v = beta == T(0) ? alpha * acc[i][j] : fma(alpha, acc[i][j], beta * *c);
                    *c = v;
                    if (sym && n < m) C[(long long)n * ldc + m] = v;
                }
            }
    }
    sc_bar(sm);
}

template <class T> struct ScTile;
template <> struct ScTile<double> { static constexpr int R = 1; };
template <> struct ScTile<float> { static constexpr int R = 2; };

template <class T>
__device__ __forceinline__ void gemm(int M, int N, int K, T alpha, const T *A, int lda, bool ta, const T *B, int ldb,
                                     bool tb, T beta, T *C, int ldc, ScShared &sm) {
    sc_gemm<T, ScTile<T>::R>(M, N, K, alpha, A, lda, ta, B, ldb, tb, beta, C, ldc, sm, false);
}

// the same for a product known to be symmetric (M == N): the tiles below the diagonal are computed
// and mirrored
template <class T>
__device__ __forceinline__ void gemm_sym(int M, int K, T alpha, const T *A, int lda, bool ta, const T *B, int ldb,
                                         bool tb, T beta, T *C, int ldc, ScShared &sm) {
    sc_gemm<T, ScTile<T>::R>(M, M, K, alpha, A, lda, ta, B, ldb, tb, beta, C, ldc, sm, true);
}

// ---------------------------------------------------------------------------------------------
// FP64 products of the iterations on the tensor cores
// ---------------------------------------------------------------------------------------------
//
// The same exact digit products as the FP64 contraction's (fixed8.cuh), on warp MMAs, so that a CTA keeps
// its registers and shared memory for the other steps: a warp computes its outputs from operands in
// digit planes, which the split writes in the order of the MMA's fragments.  An operand's rows r and its K
// elements are cut into 16 x 16 tiles (rt, kt); plane p of a tile is 32 x 16 bytes at
// [((rt nkt + kt) 8 + p) 32 + lane], lane (g, t) = (lane / 4, lane % 4) holding
// x: (row g, k 2t, 2t + 1), y: (row g, k 2t + 8, 2t + 9), z, w: the same of row g + 8: the registers of an A
// fragment of m16n8k16, and with {x, y} and {z, w} those of two B fragments, so one form serves both
// sides.  A warp's tile is 16 x 8, which leaves it the registers to have all loads of a 16-k block in
// flight; its 32 level accumulators are exact over 128 k, then folded to FP64.

// the eight planes of a lane's fixed-point values x, x, y, y, z, z, w, w
__device__ __forceinline__ void sc_store(uint4 *d, const unsigned long long (&y)[8]) {
#pragma unroll
    for (int p = 0; p < 8; ++p)
        d[p * 32] = make_uint4(cd_pair(y[0], y[1], p), cd_pair(y[2], y[3], p), cd_pair(y[4], y[5], p), cd_pair(y[6], y[7], p));
}

// digits of rows r < rows of K elements, element (r, k) at A[r * lda + k], or A[k * lda + r] when trans
__device__ __noinline__ void sc_split(const double *A, int lda, bool trans, int rows, int K, uint4 *D, int *E, const ScShared &sm) {
    const int lane = threadIdx.x & 31, nrt = (rows + 15) / 16, nkt = (K + 15) / 16;
    const int warps = SC_W * sm.csize, parts = max(1, min(warps / nrt, nkt));   // warps per row tile
    const int g = lane >> 2, t = lane & 3;
    for (int task = sm.rank * SC_W + (threadIdx.x >> 5); task < nrt * parts; task += warps) {
        const int rt = task % nrt, part = task / nrt, r0 = rt * 16;
        // bound exponents of the tile's rows, lane r: row r0 + r
        unsigned mx = 0;
        if (trans) {
            const int r = r0 + (lane & 15);
            if (r < rows)
#pragma unroll 4
                for (int k = lane >> 4; k < K; k += 2) mx = max(mx, cd_hi(A[(long long)k * lda + r]));
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        } else {
            for (int r = 0; r < 16; ++r) {
                unsigned m = 0;
                if (r0 + r < rows)
#pragma unroll 4
                    for (int k = lane; k < K; k += 32) m = max(m, cd_hi(A[(long long)(r0 + r) * lda + k]));
                m = __reduce_max_sync(0xffffffffu, m);
                if (lane == r) mx = m;
            }
        }
        const int e = cd_bound(mx);
        if (part == 0 && lane < 16) E[r0 + lane] = e;
        const int e0 = __shfl_sync(0xffffffffu, e, g), e1 = __shfl_sync(0xffffffffu, e, g + 8);
        for (int kt = part; kt < nkt; kt += parts) {
            unsigned long long y[8];   // x, x, y, y, z, z, w, w
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int r = r0 + g + (q >> 2) * 8, k = kt * 16 + 2 * t + ((q >> 1) & 1) * 8 + (q & 1);
                const int ex = (q >> 2) ? e1 : e0;
                const double v = r < rows && k < K && ex != CD_POISON
                                     ? (trans ? A[(long long)k * lda + r] : A[(long long)r * lda + k]) : 0.0;
                y[q] = cd_fixed(v, ex);
            }
            sc_store(D + ((long long)(rt * nkt + kt) * 8) * 32 + lane, y);
        }
    }
}

__device__ __forceinline__ void sc_mma(float (&c)[4], const uint4 &a, const uint2 &b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a.x), "r"(a.z), "r"(a.y), "r"(a.w), "r"(b.x), "r"(b.y));
}

// C = alpha A B^T + beta C from digits (A: M rows, B: N rows, K elements); `sym`: the tiles on and below
// the diagonal are computed and mirrored.  Returns the calling thread's part of the trace of C.
__device__ __noinline__ double sc_digit_gemm(int M, int N, int K, double alpha, const uint4 *A, const int *Ea, const uint4 *B,
                                const int *Eb, double beta, double *C, int ldc, bool sym, const ScShared &sm) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nti = (M + 15) / 16, ntj = (N + 7) / 8, nkt = (K + 15) / 16;
    const int count = sym ? nti * (nti + 1) : nti * ntj;   // sym: 2 (i + 1) column tiles in row tile i
    double trace = 0.0;
    for (int id = sm.rank * SC_W + (threadIdx.x >> 5); id < count; id += SC_W * sm.csize) {
        int ti = id / ntj, tj = id % ntj;
        if (sym) {
            ti = (int)((sqrtf(4.0f * id + 1.0f) - 1.0f) * 0.5f);
            while (ti * (ti + 1) > id) --ti;
            while ((ti + 1) * (ti + 2) <= id) ++ti;
            tj = id - ti * (ti + 1);
            if (tj >= ntj) continue;
        }
        const int e0 = Ea[ti * 16 + g], e1 = Ea[ti * 16 + g + 8];
        double out[4] = {0.0, 0.0, 0.0, 0.0};
        for (int kc = 0; kc < nkt; kc += 8) {
            float acc[8][4];   // level, fragment
#pragma unroll
            for (int l = 0; l < 8; ++l)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[l][q] = 0.0f;
            const int kend = min(kc + 8, nkt);
#pragma unroll 1
            for (int kt = kc; kt < kend; ++kt) {
                const uint4 *pa = A + ((long long)(ti * nkt + kt) * 8) * 32 + lane;
                const uint2 *pb = reinterpret_cast<const uint2 *>(B + ((long long)((tj >> 1) * nkt + kt) * 8) * 32 + lane) + (tj & 1);
                uint4 a[8];
                uint2 b[8];
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    a[p] = pa[p * 32];
                    b[p] = pb[p * 64];
                }
#pragma unroll
                for (int s = 0; s < 8; ++s)
#pragma unroll
                    for (int p = 0; p < 8 - s; ++p) sc_mma(acc[s + p], a[s], b[p]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                auto lv = [&](int l) { return (long long)__float2int_rz(acc[l][q]); };
                const long long Hs = (((lv(0) << 8) + lv(1)) << 16) + (lv(2) << 8) + lv(3);
                const long long Ls = (((lv(4) << 8) + lv(5)) << 16) + (lv(6) << 8) + lv(7);
                const int a_e = q >> 1 ? e1 : e0, b_e = Eb[tj * 8 + 2 * t + (q & 1)];
                out[q] += a_e == CD_POISON || b_e == CD_POISON ? __longlong_as_double(0x7ff8000000000000ll)
                                                               : cd_value(Hs, Ls, a_e + b_e - 68);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int m = ti * 16 + g + (q >> 1) * 8, n = tj * 8 + 2 * t + (q & 1);
            if (m < M && n < N && !(sym && n > m)) {
                double *c = C + (long long)m * ldc + n;
                const double v = beta == 0.0 ? alpha * out[q] : fma(alpha, out[q], beta * *c);
                *c = v;
                if (sym && n < m) C[(long long)n * ldc + m] = v;
                if (n == m) trace += v;
            }
        }
    }
    return trace;
}

// digit operands of a system: S and X (cut once), and the two of the running product
struct ScDig {
    uint4 *S, *X, *a, *b;
    int *eS, *eX, *ea, *eb;
};
enum ScOp { OP_S, OP_X, OP_ANY };

// whether the FP64 products of a system of n orbitals run on digits
__device__ __forceinline__ bool sc_digits(int n, const ScShared &sm) { return n * n * n >= SC_DIGITS * sm.csize; }

// A product of the iterations, C = alpha A B + beta C (A, B transposed when ta, tb): FP32 on tiles
__device__ __forceinline__ void sc_prod(const ScDig &, int M, int N, int K, float alpha, ScOp, const float *A, int lda,
                                        bool ta, ScOp, const float *B, int ldb, bool tb, float beta, float *C, int ldc,
                                        bool sym, ScShared &sm) {
    sc_gemm<float, ScTile<float>::R>(M, N, K, alpha, A, lda, ta, B, ldb, tb, beta, C, ldc, sm, sym);
}
// ... FP64 on digits, or on FP64 tiles in small systems
__device__ __noinline__ void sc_prod(const ScDig &dg, int M, int N, int K, double alpha, ScOp oa, const double *A, int lda,
                                     bool ta, ScOp ob, const double *B, int ldb, bool tb, double beta, double *C, int ldc,
                                     bool sym, ScShared &sm) {
    if (!sc_digits(max(M, K), sm)) {
        sc_gemm<double, ScTile<double>::R>(M, N, K, alpha, A, lda, ta, B, ldb, tb, beta, C, ldc, sm, sym);
        return;
    }
    const uint4 *da = oa == OP_S ? dg.S : oa == OP_X ? dg.X : dg.a, *db = ob == OP_S ? dg.S : ob == OP_X ? dg.X : dg.b;
    const int *ea = oa == OP_S ? dg.eS : oa == OP_X ? dg.eX : dg.ea, *eb = ob == OP_S ? dg.eS : ob == OP_X ? dg.eX : dg.eb;
    if (oa == OP_ANY) sc_split(A, lda, ta, M, K, dg.a, dg.ea, sm);
    if (ob == OP_ANY) {
        if (A == B && ta != tb) {   // A A^T or A^T A
            db = da;
            eb = ea;
        } else {
            sc_split(B, ldb, !tb, N, K, dg.b, dg.eb, sm);
        }
    }
    sc_bar(sm);
    sc_digit_gemm(M, N, K, alpha, da, ea, db, eb, beta, C, ldc, sym, sm);
    sc_bar(sm);
}

// ---------------------------------------------------------------------------------------------
// Symmetric eigenproblem
// ---------------------------------------------------------------------------------------------

template <class T> struct ScEps;
template <> struct ScEps<double> {
    static constexpr double eps = 2.220446049250313e-16, tiny = 2.2250738585072014e-308;
};
template <> struct ScEps<float> {
    static constexpr double eps = 1.1920928955078125e-07, tiny = 1.1754943508222875e-38;
};

// number of eigenvalues of the tridiagonal (d, squared off-diagonal esq) below x: sign changes of
// the leading principal minors N_i = (d_i - x) N_{i-1} - esq_{i-1} N_{i-2} (no division), rescaled
// by a power of two when |N_i| leaves [2^-L, 2^L]; an exact zero becomes a tiny value of the
// opposite sign
__device__ __forceinline__ int sc_sturm(const double *d, const double *esq, int n, double x) {
    double n0 = 1.0, n1 = d[0] - x;
    if (n1 == 0.0) n1 = -0x1p-100;
    int c = __double2hiint(n1) < 0;
    for (int i = 1; i < n; ++i) {
        double n2 = fma(d[i] - x, n1, -(esq[i - 1] * n0));
        const long long bits = __double_as_longlong(n2);
        if ((bits << 1) == 0) {
            n2 = -0x1p-100 * n1;
        } else {
            const int ex = (int)((bits >> 52) & 0x7ff);
            if ((ex > 1023 + 400 || ex < 1023 - 400) && ex < 2047) {
                const double s = __longlong_as_double((long long)(2046 - ex) << 52);
                n1 *= s;
                n2 *= s;
            }
        }
        c += (int)(((unsigned)__double2hiint(n1) ^ (unsigned)__double2hiint(n2)) >> 31);
        n0 = n1;
        n1 = n2;
    }
    return c;
}

__device__ __forceinline__ int sc_sturm(const float *d, const float *esq, int n, float x) {
    float n0 = 1.0f, n1 = d[0] - x;
    if (n1 == 0.0f) n1 = -0x1p-40f;
    int c = __float_as_int(n1) < 0;
    for (int i = 1; i < n; ++i) {
        float n2 = fmaf(d[i] - x, n1, -(esq[i - 1] * n0));
        const int bits = __float_as_int(n2);
        if ((bits << 1) == 0) {
            n2 = -0x1p-40f * n1;
        } else {
            const int ex = (bits >> 23) & 0xff;
            if ((ex > 127 + 40 || ex < 127 - 40) && ex < 255) {
                const float s = __int_as_float((254 - ex) << 23);   // 2^(127 - ex)
                n1 *= s;
                n2 *= s;
            }
        }
        c += (int)(((unsigned)__float_as_int(n1) ^ (unsigned)__float_as_int(n2)) >> 31);
        n0 = n1;
        n1 = n2;
    }
    return c;
}

// Lowest nr eigenpairs of the symmetric n x n matrix A (row-major, overwritten: row k keeps the
// k-th Householder vector in columns k+1..n-1).  Eigenvalues ascending into sm.w (as double),
// eigenvectors into Z [n x nr] row-major (column r = eigenvector r).  ws: 4 n nr elements, piv: n nr
// bytes.  Returns false on a non-finite value.
// CTA c of the cluster owns the rows i with i % csize = c of A in the tridiagonalisation and a
// contiguous range of the roots afterwards.  The tridiagonalisation passes one cluster barrier per
// column: before it every CTA sends its elements of p to the others' shared memory and the owner of the
// next pivot row sends that row; after it each forms the updated pivot row (and so the next
// reflection) itself.
template <class T>
__device__ bool sc_eigh(int n, int nr, T *A, T *Z, T *ws, unsigned char *piv, const ScDig &dg, ScShared &sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cs = sm.csize, rank = sm.rank;
    T *d = reinterpret_cast<T *>(sm.d), *e = reinterpret_cast<T *>(sm.e), *beta = reinterpret_cast<T *>(sm.beta);
    T *esq = reinterpret_cast<T *>(sm.esq), *u = reinterpret_cast<T *>(sm.vu), *cur = reinterpret_cast<T *>(sm.cur);
    // 1. tridiagonalisation: H_k = I - beta_k u u^T acting on rows / columns k+1..n-1; cur = row k of
    //    the reduced matrix from column k
    for (int i = tid; i < n; i += SC_T) cur[i] = A[i];
    __syncthreads();
    for (int k = 0; k + 2 < n; ++k) {
        const int n1 = n - k - 1;
        T *p = reinterpret_cast<T *>(sm.vp[k & 1]), *nxt = reinterpret_cast<T *>(sm.rb[k & 1]);
        if (warp == 0) {
            T s2 = T(0);
            for (int i = 1 + lane; i < n1; i += 32) s2 += cur[1 + i] * cur[1 + i];
            for (int off = 16; off; off >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, off);
            const T x0 = cur[1];
            T bet = T(0), alpha = x0;
            if (s2 != T(0)) {
                const T nx = sqrt(x0 * x0 + s2);
                alpha = x0 > T(0) ? -nx : nx;
                bet = T(1) / (alpha * (alpha - x0));
            }
            for (int i = 1 + lane; i < n1; i += 32) u[i] = cur[1 + i];
            if (lane == 0) {
                d[k] = cur[0];
                e[k] = alpha;
                beta[k] = bet;
                u[0] = x0 - alpha;
            }
        }
        __syncthreads();
        const T bet = beta[k];
        if (k % cs == rank)
            for (int i = tid; i < n1; i += SC_T) A[(long long)k * n + (k + 1 + i)] = u[i];
        if ((k + 1) % cs == rank)
            for (int i = tid; i < n1; i += SC_T) {
                const T v = A[(long long)(k + 1) * n + (k + 1 + i)];
                if (cs == 1) nxt[i] = v;
                else
                    for (int c = 0; c < cs; ++c) *sc_at(nxt + i, c) = v;
            }
        // own rows of the reduced matrix: first, first + cs, ...
        const int first = (rank - (k + 1) % cs + cs) % cs, own = first < n1 ? (n1 - 1 - first) / cs + 1 : 0;
        {   // p = bet A' u, G lanes per row
            const int G = n1 >= 64 ? 32 : (n1 >= 16 ? 8 : 2);
            const int rows_per_pass = SC_T / G;
            const int sub = tid % G;
            for (int base = 0; base < own; base += rows_per_pass) {   // the same trip count in every thread
                const int q = base + tid / G, r0 = first + q * cs;
                T acc = T(0);
                if (q < own) {
                    const T *ar = A + (long long)(k + 1 + r0) * n + (k + 1);
                    for (int j = sub; j < n1; j += G) acc = fma(ar[j], u[j], acc);
                }
                for (int off = G >> 1; off; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
                if (q < own) {
                    if (cs == 1) {
                        if (sub == 0) p[r0] = bet * acc;
                    } else {
                        for (int c = sub; c < cs; c += G) *sc_at(p + r0, c) = bet * acc;
                    }
                }
            }
        }
        sc_bar(sm);
        if (warp == 0) {   // q = p - (bet u.p / 2) u
            T up = T(0);
            for (int i = lane; i < n1; i += 32) up += u[i] * p[i];
            for (int off = 16; off; off >>= 1) up += __shfl_xor_sync(0xffffffffu, up, off);
            const T K = T(0.5) * bet * up;
            for (int i = lane; i < n1; i += 32) p[i] -= K * u[i];
        }
        __syncthreads();
        for (int t = tid; t < own * n1; t += SC_T) {   // A' -= u q^T + q u^T
            const int q = t / n1, i = first + q * cs, j = t - q * n1;
            T *a = A + (long long)(k + 1 + i) * n + (k + 1 + j);
            *a = fma(-u[i], p[j], fma(-p[i], u[j], *a));
        }
        for (int j = tid; j < n1; j += SC_T) cur[j] = fma(-u[0], p[j], fma(-p[0], u[j], nxt[j]));
        __syncthreads();
    }
    sc_bar(sm);   // the last row and every Householder vector
    if (tid == 0) {
        d[n - 2] = cur[0];
        e[n - 2] = cur[1];
        beta[n - 2] = T(0);
        d[n - 1] = A[(long long)(n - 1) * n + n - 1];
        e[n - 1] = T(0);
        beta[n - 1] = T(0);
    }
    __syncthreads();
    // 2. Gershgorin interval, e^2, finiteness
    double glo = 1e300, ghi = -1e300, emax2 = 0.0;
    bool fin = true;
    for (int i = tid; i < n; i += SC_T) {
        const double r = fabs((double)e[i]) + (i > 0 ? fabs((double)e[i - 1]) : 0.0);
        glo = fmin(glo, (double)d[i] - r);
        ghi = fmax(ghi, (double)d[i] + r);
        esq[i] = e[i] * e[i];
        emax2 = fmax(emax2, (double)esq[i]);
        fin = fin && isfinite((double)d[i]) && isfinite((double)e[i]);
    }
    glo = -sc_max_cta(-glo, sm);
    ghi = sc_max_cta(ghi, sm);
    emax2 = sc_max_cta(emax2, sm);
    if (sc_max_cta(fin ? 0.0 : 1.0, sm) != 0.0) return false;   // the same in every CTA
    const double eps = ScEps<T>::eps;
    const double tnorm = fmax(fabs(glo), fabs(ghi));
    const double pivmin = ScEps<T>::tiny * fmax(1.0, emax2) * 4.0;
    const int chunk = (nr + cs - 1) / cs, rbeg = min(rank * chunk, nr), nc = min(chunk, nr - rbeg);   // own roots
    // 3. eigenvalues by multisection on Sturm counts: P lanes per root take P points of its interval
    //    (an FP64 warp instruction costs the same for one lane as for 32), as many as keep one warp per
    //    sub-partition; P = 1 is bisection with one thread per root
    int P = 1;
    while (P < 32 && 2 * P * chunk <= 128) P *= 2;
    for (int base = 0; base < nc * P; base += SC_T) {   // the same trip count in every thread
        const int id = base + tid, r = rbeg + id / P, j = id % P;
        bool active = id < nc * P;
        const unsigned group = (P == 32 ? 0xffffffffu : ((1u << P) - 1u) << (lane & ~(P - 1)));
        T a = (T)(glo - (2.0 * eps * tnorm + 2.0 * pivmin)), b = (T)(ghi + (2.0 * eps * tnorm + 2.0 * pivmin));
        for (int it = 0; it < 80 && __any_sync(0xffffffffu, active); ++it) {
            const T mag = fmax(fabs(a), fabs(b));
            // bisection near the end, where the points would fall on neighbouring numbers
            const bool bis = P == 1 || !(b - a > T(64.0 * eps) * mag);
            const T h = (b - a) / T(P + 1);
            auto point = [&](int i) { return bis ? T(0.5) * (a + b) : a + T(i + 1) * h; };
            const T x = point(j);
            if (!(b - a > T(2.0 * eps) * mag + T(pivmin)) || x <= a || x >= b) active = false;
            const bool above = active && sc_sturm(d, esq, n, x) > r;
            const unsigned m = (__ballot_sync(0xffffffffu, above) & group) >> (lane & ~(P - 1));
            if (active) {
                const int f = m ? __ffs(m) - 1 : P;   // first point above the root
                const T na = f > 0 ? point(f - 1) : a, nb = f < P ? point(f) : b;
                a = na;
                b = nb;
            }
        }
        if (id < nc * P && j == 0) {
            const double w = 0.5 * ((double)a + (double)b);
            if (cs == 1) sm.w[r] = w;
            else
                for (int c = 0; c < cs; ++c) *sc_at(&sm.w[r], c) = w;
        }
    }
    sc_bar(sm);
    // 4. inverse iteration, one thread per root: LU of T - w_r I with partial pivoting (factors
    //    interleaved over the roots, [i * nr + r], so a warp's accesses are contiguous), then three
    //    solves from a fixed start vector; the recurrences run in registers
    const T tiny = (T)(eps * fmax(tnorm, 1e-30));
    for (int r = rbeg + tid; r < rbeg + nc; r += SC_T) {
        const T lam = (T)sm.w[r];
        T *__restrict__ DL = ws;
        T *__restrict__ DD = ws + (long long)n * nr;
        T *__restrict__ DU = ws + 2LL * n * nr;
        T *__restrict__ DU2 = ws + 3LL * n * nr;
        unsigned char *__restrict__ PV = piv;
        T *__restrict__ Zr = Z;
#define IX(i) ((long long)(i) * nr + r)
        T cdd = d[0] - lam, cdu = e[0];
        for (int i = 0; i + 1 < n; ++i) {
            const T li = e[i], dn = d[i + 1] - lam, un = e[i + 1];
            if (fabs(cdd) >= fabs(li)) {
                const T dv = fabs(cdd) < tiny ? (cdd < T(0) ? -tiny : tiny) : cdd;
                const T rp = T(1) / dv, l = li * rp;
                DD[IX(i)] = rp;
                DL[IX(i)] = l;
                DU[IX(i)] = cdu;
                DU2[IX(i)] = T(0);
                PV[IX(i)] = 0;
                cdd = dn - l * cdu;
                cdu = un;
            } else {
                const T rp = T(1) / li, l = cdd * rp;
                DD[IX(i)] = rp;
                DL[IX(i)] = l;
                DU[IX(i)] = dn;
                DU2[IX(i)] = i + 2 < n ? un : T(0);
                PV[IX(i)] = 1;
                cdd = cdu - l * dn;
                cdu = -l * un;
            }
        }
        DD[IX(n - 1)] = T(1) / (fabs(cdd) < tiny ? (cdd < T(0) ? -tiny : tiny) : cdd);
        DU[IX(n - 1)] = T(0);
        DU2[IX(n - 1)] = T(0);
        for (int it = 0; it < 3; ++it) {
            // L^-1 with the interchanges (the start vector is generated in the first pass)
            auto start = [&](int i) { return T(1) + T(0.5) * (T)((i * (r + 1) * 7919 + 13 * r) % 97) / T(97); };
            T zc = it == 0 ? start(0) : Zr[IX(0)];
#pragma unroll 4
            for (int i = 0; i + 1 < n; ++i) {
                T zn = it == 0 ? start(i + 1) : Zr[IX(i + 1)];
                if (PV[IX(i)]) { const T t = zc; zc = zn; zn = t; }
                zn -= DL[IX(i)] * zc;
                Zr[IX(i)] = zc;
                zc = zn;
            }
            Zr[IX(n - 1)] = zc;
            // U^-1 and the norm
            T z1 = T(0), z2 = T(0), nrm = T(0);
#pragma unroll 4
            for (int i = n - 1; i >= 0; --i) {
                T v = Zr[IX(i)] - DU[IX(i)] * z1 - DU2[IX(i)] * z2;
                v *= DD[IX(i)];
                Zr[IX(i)] = v;
                nrm = fma(v, v, nrm);
                z2 = z1;
                z1 = v;
            }
            nrm = T(1) / sqrt(nrm);
#pragma unroll 4
            for (int i = 0; i < n; ++i) Zr[IX(i)] *= nrm;
        }
#undef IX
    }
    sc_bar(sm);
    // 5. orthonormalisation.  Inverse iteration leaves overlaps of order eps |T| / gap, so Z^T Z = I + D with
    //    a tiny D unless roots (nearly) coincide, and Z (I - D / 2) is orthonormal to D^2 (Loewdin's
    //    orthogonalisation to first order): two products instead of a chain of Gram-Schmidt steps along
    //    clusters that take in most of the spectrum at LAPACK dstein's 1e-3 |T|.  With overlaps of 1e-8 and
    //    more: Gram-Schmidt (twice) inside clusters of roots closer than 1e-3 |T|, one warp per cluster.
    T *D = ws, *Z2 = ws + (long long)nr * nr;
    sc_prod(dg, nr, nr, n, T(1), OP_ANY, Z, nr, true, OP_ANY, Z, nr, false, T(0), D, nr, true, sm);
    double dmax = 0.0;
    SC_FOR(t, (long long)nr * nr) {
        const int i = (int)(t / nr), j = (int)(t - (long long)i * nr);
        const T v = (i == j ? T(1) : T(0)) - D[t];
        dmax = fmax(dmax, fabs((double)v));
        D[t] = T(0.5) * v;
    }
    dmax = sc_max(dmax, sm);
    if (dmax < (sizeof(T) == 8 ? 1e-8 : 1e-4)) {
        sc_bar(sm);
        sc_prod(dg, n, nr, nr, T(1), OP_ANY, Z, nr, false, OP_ANY, D, nr, false, T(0), Z2, nr, false, sm);
        SC_FOR(t, (long long)n * nr) Z[t] += Z2[t];
    } else {
        const double ortol = 1e-3 * tnorm;
        int c0 = 0, id = 0;
        for (int r = 1; r < nr; ++r) {
            if (sm.w[r] - sm.w[r - 1] > ortol) {
                c0 = r;
                ++id;
                continue;
            }
            if (id % (SC_W * cs) != rank * SC_W + warp) continue;
            // root r in registers, row lane + 32 q in z[q]; its predecessors stream through
            T z[SC_NMAX / 32], y[SC_NMAX / 32];
            auto read = [&](int root, T (&x)[SC_NMAX / 32]) {
#pragma unroll
                for (int q = 0; q < SC_NMAX / 32; ++q)
                    x[q] = lane + 32 * q < n ? Z[(long long)(lane + 32 * q) * nr + root] : T(0);
            };
            read(r, z);
            for (int pass = 0; pass < 2; ++pass)
                for (int p = c0; p < r; ++p) {
                    read(p, y);
                    T dot = T(0);
#pragma unroll
                    for (int q = 0; q < SC_NMAX / 32; ++q)
                        if (32 * q < n) dot = fma(y[q], z[q], dot);
                    for (int off = 16; off; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
#pragma unroll
                    for (int q = 0; q < SC_NMAX / 32; ++q)
                        if (32 * q < n) z[q] = fma(-dot, y[q], z[q]);
                }
            T nrm = T(0);
#pragma unroll
            for (int q = 0; q < SC_NMAX / 32; ++q)
                if (32 * q < n) nrm = fma(z[q], z[q], nrm);
            for (int off = 16; off; off >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, off);
            nrm = T(1) / sqrt(nrm);
#pragma unroll
            for (int q = 0; q < SC_NMAX / 32; ++q)
                if (lane + 32 * q < n) Z[(long long)(lane + 32 * q) * nr + r] = z[q] * nrm;
        }
    }
    sc_bar(sm);
    // 6. back-transformation Z <- H_0 ... H_{n-3} Z of the own columns (no exchange between CTAs)
    if (chunk <= 2 * SC_W) {
        // few columns: two per warp in registers, row lane + 32 q in z[q]
        const int r0 = rbeg + warp, r1 = r0 + SC_W;
        const bool h0 = warp < nc, h1 = warp + SC_W < nc;
        T z0[SC_NMAX / 32], z1[SC_NMAX / 32];
#pragma unroll
        for (int q = 0; q < SC_NMAX / 32; ++q) {
            const int i = lane + 32 * q;
            z0[q] = h0 && i < n ? Z[(long long)i * nr + r0] : T(0);
            z1[q] = h1 && i < n ? Z[(long long)i * nr + r1] : T(0);
        }
        if (h0)
            for (int k = n - 3; k >= 0; --k) {
                const T bet = beta[k];
                if (bet == T(0)) continue;
                T uk[SC_NMAX / 32], s0 = T(0), s1 = T(0);
#pragma unroll
                for (int q = 0; q < SC_NMAX / 32; ++q) {
                    const int i = lane + 32 * q;
                    if (32 * q + 31 <= k || 32 * q >= n) continue;   // the same in every lane
                    uk[q] = i > k && i < n ? A[(long long)k * n + i] : T(0);
                    s0 = fma(uk[q], z0[q], s0);
                    if (h1) s1 = fma(uk[q], z1[q], s1);
                }
                for (int off = 16; off; off >>= 1) {
                    s0 += __shfl_xor_sync(0xffffffffu, s0, off);
                    if (h1) s1 += __shfl_xor_sync(0xffffffffu, s1, off);
                }
                s0 *= -bet;
                s1 *= -bet;
#pragma unroll
                for (int q = 0; q < SC_NMAX / 32; ++q) {
                    if (32 * q + 31 <= k || 32 * q >= n) continue;
                    z0[q] = fma(s0, uk[q], z0[q]);
                    if (h1) z1[q] = fma(s1, uk[q], z1[q]);
                }
            }
#pragma unroll
        for (int q = 0; q < SC_NMAX / 32; ++q) {
            const int i = lane + 32 * q;
            if (h0 && i < n) Z[(long long)i * nr + r0] = z0[q];
            if (h1 && i < n) Z[(long long)i * nr + r1] = z1[q];
        }
    } else {
        // `sub` threads per column, each with the rows i = sb (mod sub); the dots' parts alternate
        // between two buffers, so one barrier per reflection
        const int ncp = (nc + 31) / 32 * 32, sub = ncp > 0 ? SC_T / ncp : 1, c = ncp > 0 ? tid % ncp : 0;
        const int sb = ncp > 0 ? tid / ncp : 0;
        const bool on = c < nc && sb < sub;
        T *Zc = Z + rbeg + c;
        int buf = 0;
        for (int k = n - 3; k >= 0; --k) {
            const T bet = beta[k];
            if (bet == T(0)) continue;
            T *part = reinterpret_cast<T *>(sm.gemm) + buf * SC_T;
            buf ^= 1;
            const T *uk = A + (long long)k * n;
            const int i0 = k + 1 + ((sb - (k + 1)) % sub + sub) % sub;
            T acc = T(0);
            if (on)
#pragma unroll 4
                for (int i = i0; i < n; i += sub) acc = fma(uk[i], Zc[(long long)i * nr], acc);
            part[tid] = acc;
            __syncthreads();
            if (on) {
                T v = T(0);
                for (int q = 0; q < sub; ++q) v += part[q * ncp + c];
                v *= -bet;
#pragma unroll 4
                for (int i = i0; i < n; i += sub) Zc[(long long)i * nr] = fma(v, uk[i], Zc[(long long)i * nr]);
            }
        }
    }
    sc_bar(sm);
    return true;
}

// ---------------------------------------------------------------------------------------------
// per-slot storage
// ---------------------------------------------------------------------------------------------

// FP64 inputs of the current system (S, H0, X = S^-1/2, Sh = S^1/2, gamma, gamma_lr, reference
// occupations p0) followed by the work area (29 n^2 doubles), used as T elements by the phase that
// runs (the FP32 phase keeps FP32 copies of the inputs in it), and the pivot flags (n^2 bytes).
struct ScSlot {
    double *S, *H0, *X, *Sh, *gam, *glr, *p0;
    unsigned char *work;
    unsigned char *piv;
    ScDig dg;
};

constexpr int SC_WORK = 29;   // n x n blocks of the work area

__host__ __device__ inline long long sc_slot_doubles(long long nn, long long at2, long long npad) {
    return 4 * nn + 2 * at2 + npad + SC_WORK * nn;
}

// bytes of the digit operands of a slot for np (a multiple of 16) orbitals, a multiple of 256
__host__ __device__ inline long long sc_digit_bytes(long long np) {
    return (4 * np * np * 16 + 4 * np * 4 + 255) / 256 * 256;
}

__device__ ScSlot sc_slot(const ScArgs &a, int slot) {
    double *f = reinterpret_cast<double *>(a.ws + (long long)slot * a.slot_bytes);
    ScSlot s;
    s.S = f;
    s.H0 = f + a.nn_max;
    s.X = f + 2 * a.nn_max;
    s.Sh = f + 3 * a.nn_max;
    s.gam = f + 4 * a.nn_max;
    s.glr = s.gam + a.at2_max;
    s.p0 = s.glr + a.at2_max;
    s.work = reinterpret_cast<unsigned char *>(s.p0 + a.npad);
    s.piv = s.work + SC_WORK * a.nn_max * (long long)sizeof(double);
    // digit planes (16-byte aligned): 16 bytes per element of 16 x 16 tiles, then the rows' exponents
    const long long np = (a.npad + 15) / 16 * 16, per = np * np;
    uint4 *d = reinterpret_cast<uint4 *>(a.ws + (long long)(slot + 1) * a.slot_bytes - sc_digit_bytes(np));
    s.dg.S = d;
    s.dg.X = d + per;
    s.dg.a = d + 2 * per;
    s.dg.b = d + 3 * per;
    int *e = reinterpret_cast<int *>(d + 4 * per);
    s.dg.eS = e;
    s.dg.eX = e + np;
    s.dg.ea = e + 2 * np;
    s.dg.eb = e + 3 * np;
    return s;
}

template <class T> struct ScWork {
    T *S, *H0, *X, *Sh, *gam, *glr;     // inputs in T (FP64: the slot's arrays)
    T *F, *Fp, *P, *Pp, *T1, *T2, *T3, *EA, *Z, *W;   // n x n each (W: 4 n x n)
    T *Fh, *Eh;                         // SC_DIIS n x n each
    ScDig dg;
};

template <class T>
__device__ ScWork<T> sc_work(const ScSlot &s, long long nn) {
    ScWork<T> w;
    T *b = reinterpret_cast<T *>(s.work);
    w.F = b; w.Fp = b + nn; w.P = b + 2 * nn; w.Pp = b + 3 * nn; w.T1 = b + 4 * nn; w.T2 = b + 5 * nn;
    w.T3 = b + 6 * nn; w.EA = b + 7 * nn; w.Z = b + 8 * nn; w.W = b + 9 * nn;
    w.Fh = b + 13 * nn; w.Eh = b + (13 + SC_DIIS) * nn;
    w.dg = s.dg;
    return w;
}

// ---------------------------------------------------------------------------------------------
// system set-up: AO tables, S, H0, gamma, gamma_lr, repulsion (FP64)
// ---------------------------------------------------------------------------------------------

__device__ double sc_setup(const ScArgs &a, const tincr_scc_system &sy, const ScSlot &sl, ScShared &sm) {
    const int tid = threadIdx.x, N = sy.n_atoms, n = sy.n_orb;
    const int *kind = a.kind + sy.atom_off;
    const double *xyz = a.xyz + 3 * sy.atom_off;
    for (int A = tid; A < N; A += SC_T) sm.kind[A] = kind[A];
    __syncthreads();
    if (tid == 0) {
        int o = 0;
        for (int A = 0; A < N; ++A) {
            sm.ao_off[A] = o;
            o += a.kind_norb[sm.kind[A]];
        }
        sm.ao_off[N] = o;
    }
    __syncthreads();
    for (int A = tid; A < N; A += SC_T)
        for (int mu = sm.ao_off[A]; mu < sm.ao_off[A + 1]; ++mu) sm.ao_atom[mu] = (short)A;
    __syncthreads();
    const long long nn = (long long)n * n;
    SC_FOR(t, nn) {
        const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
        double sv = 0.0, hv = 0.0;
        if (mu == nu) {
            const int A = sm.ao_atom[mu];
            sv = 1.0;
            hv = a.kind_energy[4 * sm.kind[A] + (mu - sm.ao_off[A])];
        }
        sl.S[t] = a.s_in ? a.s_in[sy.mat_off + t] : sv;
        sl.H0[t] = a.h0_in ? a.h0_in[sy.mat_off + t] : hv;
    }
    sc_bar(sm);
    const bool build_sk = !a.s_in || !a.h0_in;
    // atom pairs A < B
    double erep = 0.0;
    SC_FOR(t, N * N) {
        const int A = (int)(t / N), B = (int)(t - (long long)A * N);
        const int kA = sm.kind[A], kB = sm.kind[B];
        const double dx = xyz[3 * B] - xyz[3 * A], dy = xyz[3 * B + 1] - xyz[3 * A + 1], dz = xyz[3 * B + 2] - xyz[3 * A + 2];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        // gamma (gamma_approximation.rs:75-124, diagonal :175-193)
        {
            const double sA = a.sigma[kA], sB = a.sigma[kB];
            double g, gl = 0.0;
            if (A == B) {
                g = 1.0 / sqrt(3.141592653589793 * sA * sA);
                if (a.lc) gl = 1.0 / sqrt(3.141592653589793 * (sA * sA + 0.25 * a.r_lr * a.r_lr));
            } else {
                g = erf(r / sqrt(2.0 * (sA * sA + sB * sB))) / r;
                if (a.lc) gl = erf(r / sqrt(2.0 * (sA * sA + sB * sB + 0.5 * a.r_lr * a.r_lr))) / r;
            }
            sl.gam[t] = a.gam_in ? a.gam_in[sy.pair_off + t] : g;
            sl.glr[t] = a.lc ? (a.glr_in ? a.glr_in[sy.pair_off + t] : gl) : 0.0;
        }
        if (A >= B) continue;
        // repulsion (pairs within the spline's range)
        if (a.rep_nt) {
            const int pk = kA * a.n_kinds + kB;
            if (r <= a.rep_dmax[pk]) {
                int l;
                double N3[4], N2[3], v = 0.0, dv;
                const double *tk = a.rep_knots + (long long)pk * a.rep_ntmax;
                if (bspline3_basis(tk, a.rep_nt[pk], r, l, N3, N2))
                    bspline3_eval(tk, a.rep_coef + (long long)pk * a.rep_ntmax, l, N3, N2, v, dv);
                erep += v;
            }
        }
        // Slater-Koster block: centre 1 the lower Z, ties by index (h0_and_s.rs:92-182)
        if (!build_sk || r >= SC_PROXIMITY) continue;
        const bool swap = a.kind_z[kA] > a.kind_z[kB];
        const int c1 = swap ? B : A, c2 = swap ? A : B;
        const int k1 = sm.kind[c1], k2 = sm.kind[c2];
        const double sg = swap ? -1.0 : 1.0;
        const double u[3] = {sg * dx / r, sg * dy / r, sg * dz / r};
        double vS[SK_SLOTS] = {0, 0, 0, 0, 0}, vH[SK_SLOTS] = {0, 0, 0, 0, 0}, dS[SK_SLOTS], dH[SK_SLOTS];
        int l;
        double N3[4], N2[3];
        if (bspline3_basis(a.knots, a.n_knots, r, l, N3, N2, a.sk_extrapolate != 0)) {
            const double *cS = a.coef + (long long)((k1 * a.n_kinds + k2) * 2 + 0) * SK_SLOTS * a.n_knots;
            const double *cH = a.coef + (long long)((k1 * a.n_kinds + k2) * 2 + 1) * SK_SLOTS * a.n_knots;
            for (int q = 0; q < SK_SLOTS; ++q) {
                bspline3_eval(a.knots, cS + (long long)q * a.n_knots, l, N3, N2, vS[q], dS[q]);
                bspline3_eval(a.knots, cH + (long long)q * a.n_knots, l, N3, N2, vH[q], dH[q]);
            }
        }
        const int n1 = a.kind_norb[k1], n2 = a.kind_norb[k2];
        for (int pp = 0; pp < n1; ++pp)
            for (int qq = 0; qq < n2; ++qq) {
                const int l1 = a.kind_l[4 * k1 + pp], m1 = a.kind_m[4 * k1 + pp];
                const int l2 = a.kind_l[4 * k2 + qq], m2 = a.kind_m[4 * k2 + qq];
                const double sv = sk_value(l1, m1, l2, m2, u, vS), hv = sk_value(l1, m1, l2, m2, u, vH);
                const int mu = sm.ao_off[c1] + pp, nu = sm.ao_off[c2] + qq;
                if (!a.s_in) {
                    sl.S[(long long)mu * n + nu] = sv;
                    sl.S[(long long)nu * n + mu] = sv;
                }
                if (!a.h0_in) {
                    sl.H0[(long long)mu * n + nu] = hv;
                    sl.H0[(long long)nu * n + mu] = hv;
                }
            }
    }
    const double e = sc_sum(erep, sm);
    sc_bar(sm);
    return e;
}

// ---------------------------------------------------------------------------------------------
// SCC pieces
// ---------------------------------------------------------------------------------------------

// Mulliken charge differences of dP = P - diag(p0) into sm.dq (double), esp = gamma dq into sm.esp
template <class T>
__device__ void sc_charges(int n, int N, const T *P, const T *S, const T *gam, const double *p0, ScShared &sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int mu = sm.rank * SC_W + warp; mu < n; mu += SC_W * sm.csize) {
        T acc = T(0);
        const T *pr = P + (long long)mu * n, *sr = S + (long long)mu * n;
        for (int nu = lane; nu < n; nu += 32) acc = fma(pr[nu], sr[nu], acc);
        for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        const double q = (double)acc - p0[mu];   // S_mumu = 1
        if (sm.csize == 1) {
            if (lane == 0) sm.qao[mu] = q;
        } else if (lane < sm.csize) {
            *sc_at(&sm.qao[mu], lane) = q;
        }
    }
    sc_bar(sm);
    for (int A = tid; A < N; A += SC_T) {
        double q = 0.0;
        for (int mu = sm.ao_off[A]; mu < sm.ao_off[A + 1]; ++mu) q += sm.qao[mu];
        sm.dq[A] = q;
    }
    __syncthreads();
    for (int A = tid; A < N; A += SC_T) {
        double s = 0.0;
        for (int B = 0; B < N; ++B) s = fma((double)gam[(long long)A * N + B], sm.dq[B], s);
        sm.esp[A] = s;
    }
    __syncthreads();
}

// F = H0 + 1/2 S o (esp_mu + esp_nu) [+ H^x(dP)]  (scc_routine.rs:176-183; helpers.rs:111-155)
template <class T>
__device__ void sc_fock(int n, int N, bool lc, const ScWork<T> &w, const double *p0, ScShared &sm) {
    const long long nn = (long long)n * n;
    SC_FOR(t, nn) {
        const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
        const T es = (T)(0.5 * (sm.esp[sm.ao_atom[mu]] + sm.esp[sm.ao_atom[nu]]));
        w.F[t] = fma(es, w.S[t], w.H0[t]);
    }
    if (!lc) {
        sc_bar(sm);
        return;
    }
    T *dP = w.W, *hx = w.W + nn, *tmp = w.W + 2 * nn;
    SC_FOR(t, nn) {
        const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
        dP[t] = w.P[t] - (mu == nu ? (T)p0[mu] : T(0));
    }
    sc_bar(sm);
#define GLR(mu, nu) w.glr[(long long)sm.ao_atom[mu] * N + sm.ao_atom[nu]]
    sc_prod(w.dg, n, n, n, T(1), OP_S, w.S, n, false, OP_ANY, dP, n, false, T(0), w.T1, n, false, sm);   // S dP
    SC_FOR(t, nn) {
        const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
        tmp[t] = GLR(mu, nu) * w.T1[t];
    }
    sc_bar(sm);
    sc_prod(w.dg, n, n, n, T(1), OP_ANY, tmp, n, false, OP_S, w.S, n, false, T(0), w.T2, n, false, sm);   // (g o S dP) S
    sc_prod(w.dg, n, n, n, T(1), OP_ANY, w.T1, n, false, OP_S, w.S, n, false, T(0), w.T3, n, true, sm);   // S dP S
    SC_FOR(t, nn) {
        const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
        const T g = GLR(mu, nu);
        hx[t] = w.T2[t] + w.T2[(long long)nu * n + mu] + g * w.T3[t];
        tmp[t] = dP[t] * g;
    }
    sc_bar(sm);
    sc_prod(w.dg, n, n, n, T(1), OP_S, w.S, n, false, OP_ANY, tmp, n, false, T(0), w.T1, n, false, sm);   // S (dP o g)
    sc_prod(w.dg, n, n, n, T(1), OP_ANY, w.T1, n, false, OP_S, w.S, n, false, T(1), hx, n, true, sm);    // + S (dP o g) S
    SC_FOR(t, nn) {
        const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
        w.F[t] += T(-0.0625) * (hx[t] + hx[(long long)nu * n + mu]);
    }
#undef GLR
    sc_bar(sm);
}

// solve the DIIS equations (m + 1 unknowns, the last the multiplier) on thread 0; sm.coef
__device__ void sc_diis_solve(int m, int cur, ScShared &sm) {
    if (threadIdx.x == 0) {
        const int q = m + 1, ld = q + 1;
        double *L = sm.lin;
        for (int i = 0; i < q; ++i) {
            for (int j = 0; j < q; ++j) L[i * ld + j] = (i < m && j < m) ? sm.B[i][j] : (i == m && j == m ? 0.0 : -1.0);
            L[i * ld + q] = i == m ? -1.0 : 0.0;
        }
        bool ok = true;
        for (int c = 0; c < q && ok; ++c) {
            int pr = c;
            for (int i = c + 1; i < q; ++i)
                if (fabs(L[i * ld + c]) > fabs(L[pr * ld + c])) pr = i;
            if (!(fabs(L[pr * ld + c]) > 0.0)) { ok = false; break; }
            if (pr != c)
                for (int j = 0; j <= q; ++j) { const double t = L[c * ld + j]; L[c * ld + j] = L[pr * ld + j]; L[pr * ld + j] = t; }
            for (int i = c + 1; i < q; ++i) {
                const double f = L[i * ld + c] / L[c * ld + c];
                for (int j = c; j <= q; ++j) L[i * ld + j] -= f * L[c * ld + j];
            }
        }
        if (ok) {
            for (int i = q - 1; i >= 0; --i) {
                double v = L[i * ld + q];
                for (int j = i + 1; j < q; ++j) v -= L[i * ld + j] * sm.coef[j];
                sm.coef[i] = v / L[i * ld + i];
            }
            for (int i = 0; i < m; ++i) ok = ok && isfinite(sm.coef[i]);
        }
        if (!ok)
            for (int i = 0; i < m; ++i) sm.coef[i] = i == cur ? 1.0 : 0.0;
    }
    __syncthreads();
}

// Density of the o lowest states of the symmetric matrix F without its eigenpairs: X ends as the projector
// onto them.  Trace-correcting purification (Niklasson, Phys. Rev. B 66, 155115 (2002)): X_0 maps the
// spectrum into [0, 1] with the lowest states near 1, and each step takes X^2 or 2 X - X^2, whichever
// brings the trace closer to o, until X = X^2.  Some twenty-five symmetric products, which run on digits,
// in place of a tridiagonal eigenproblem bound by FP64 latency.  The elements of X stay within [-1, 1],
// so its digits need no row maxima and are cut by the pass that updates X.  False (X undefined) when the
// spectrum has no gap there that 60 steps resolve, or is not finite; the caller then diagonalises.
// Y: n x n of work.
__device__ __noinline__ bool sc_purify(int n, int o, const double *F, double *X, double *Y, const ScDig &dg, ScShared &sm) {
    const int lane = threadIdx.x & 31, gw = sm.rank * SC_W + (threadIdx.x >> 5), warps = SC_W * sm.csize;
    double lo = 1e300, hi = -1e300;   // Gershgorin bounds
    for (int i = gw; i < n; i += warps) {
        double r = 0.0;
        for (int j = lane; j < n; j += 32) r += j == i ? 0.0 : fabs(F[(long long)i * n + j]);
        for (int off = 16; off; off >>= 1) r += __shfl_xor_sync(0xffffffffu, r, off);
        const double d = F[(long long)i * n + i];
        lo = fmin(lo, d - r);
        hi = isfinite(d) && isfinite(r) ? fmax(hi, d + r) : HUGE_VAL;   // fmin and fmax drop a NaN
    }
    lo = -sc_max(-lo, sm);
    hi = sc_max(hi, sm);
    const double w = hi - lo;
    if (!(w > 0.0) || !isfinite(w)) return false;   // the same in every thread of the cluster
    const double s = 1.0 / w;
    const bool dig = sc_digits(n, sm);
    const int nt = (n + 15) / 16, g = lane >> 2, t = lane & 3;
    // X = X_0 (mode 0), Y (1) or 2 X - Y (2), with its digits
    auto update = [&](int mode) {
        auto value = [&](int r, int k) {
            const long long x = (long long)r * n + k;
            const double v = mode == 0 ? s * ((r == k ? hi : 0.0) - F[x]) : mode == 1 ? Y[x] : 2.0 * X[x] - Y[x];
            X[x] = v;
            return v;
        };
        if (dig) {
            for (int task = gw; task < nt * nt; task += warps) {
                const int rt = task / nt, kt = task % nt;
                unsigned long long y[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int r = rt * 16 + g + (q >> 2) * 8, k = kt * 16 + 2 * t + ((q >> 1) & 1) * 8 + (q & 1);
                    y[q] = cd_fixed(r < n && k < n ? value(r, k) : 0.0, 0);
                }
                sc_store(dg.a + ((long long)task * 8) * 32 + lane, y);
            }
        } else {
            SC_FOR(x, (long long)n * n) value((int)(x / n), (int)(x % n));
        }
        sc_bar(sm);
    };
    if (dig) SC_FOR(r, nt * 16) dg.ea[r] = 0;
    update(0);
    double t1 = 0.0;
    SC_FOR(i, n) t1 += X[i * n + i];
    t1 = sc_sum(t1, sm);
    bool prev = false, last = false;
    for (int it = 0; it < 60; ++it) {
        double t2 = 0.0;   // Y = X^2 and its trace
        if (dig) {
            t2 = sc_digit_gemm(n, n, n, 1.0, dg.a, dg.ea, dg.a, dg.ea, 0.0, Y, n, true, sm);
        } else {
            sc_gemm<double, ScTile<double>::R>(n, n, n, 1.0, X, n, false, X, n, true, 0.0, Y, n, sm, true);
            SC_FOR(i, n) t2 += Y[i * n + i];
        }
        t2 = sc_sum(t2, sm);
        if (sm.csize == 1) __syncthreads();
        if (!isfinite(t2)) return false;
        // the last step is the other one: eigenvalues off by d from 0 and from 1 are then both off by d^2
        const bool square = last ? !prev : fabs(t2 - o) <= fabs(2.0 * t1 - t2 - o);
        const bool near = fabs(t1 - t2) < 1e-8;
        update(square ? 1 : 2);
        t1 = square ? t2 : 2.0 * t1 - t2;
        if (last) return fabs(t1 - o) < 1e-7;
        last = near;
        prev = square;
    }
    return false;
}

struct ScState {
    int it;            // iterations done (both phases)
    bool converged;
    double errn;
    bool finite;
};

// SCC iterations in arithmetic T from the AO density in w.P: at most `limit` iterations; stops when
// the commutator is below `stop` (after at least one diagonalisation in total).  On return w.F and
// w.Fp hold the Fock matrix of the last iterate (from its density) and st.errn its commutator.
// `hist`: DIIS entries so far (in w.Fh / w.Eh and sm.B); the entry of the last iterate is stored in
// slot hist % SC_DIIS but not counted, so the next phase's first iterate replaces it.
template <class T>
__device__ void sc_iterate(const ScArgs &a, const tincr_scc_system &sy, const ScWork<T> &w, unsigned char *piv,
                           const double *p0, int limit, double stop, ScState &st, int &hist, ScShared &sm) {
    const int tid = threadIdx.x, n = sy.n_orb, N = sy.n_atoms, o = sy.n_occ;
    const long long nn = (long long)n * n;
    // P' = S^1/2 P S^1/2 of the starting density
    gemm<T>(n, n, n, T(1), w.Sh, n, false, w.P, n, false, T(0), w.T1, n, sm);
    gemm_sym<T>(n, n, T(1), w.T1, n, false, w.Sh, n, false, T(0), w.Pp, n, sm);
    // a matrix without a gap costs all steps of the purification and the eigenpairs too, and often stays so: after
    // each failure in a row twice as many iterations (32 at most) go to the eigenpairs at once (77 stacked
    // anthracene dimers without LC, three of which never converge: 1357 -> 873 ms, 2047 with the eigenpairs alone)
    int failed = 0, wait = 0;
    for (int k = 0; k < limit; ++k) {
        ++st.it;
        sc_charges<T>(n, N, w.P, w.S, w.gam, p0, sm);
        sc_fock<T>(n, N, a.lc != 0, w, p0, sm);
        // F' = X F X, E' = F' P' - P' F'
        sc_prod(w.dg, n, n, n, T(1), OP_X, w.X, n, false, OP_ANY, w.F, n, false, T(0), w.T1, n, false, sm);
        sc_prod(w.dg, n, n, n, T(1), OP_ANY, w.T1, n, false, OP_X, w.X, n, false, T(0), w.Fp, n, true, sm);
        sc_prod(w.dg, n, n, n, T(1), OP_ANY, w.Fp, n, false, OP_ANY, w.Pp, n, false, T(0), w.T1, n, false, sm);
        const int cur = hist % SC_DIIS;
        T *Fc = w.Fh + cur * nn, *Ec = w.Eh + cur * nn;
        double emax = 0.0;
        bool fin = true;
        SC_FOR(t, nn) {
            const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
            const T ev = w.T1[t] - w.T1[(long long)nu * n + mu];
            Ec[t] = ev;
            Fc[t] = w.Fp[t];
            emax = fmax(emax, fabs((double)ev));
            fin = fin && isfinite((double)w.Fp[t]);
        }
        st.errn = sc_max(emax, sm);
        if (sc_max(fin && isfinite(st.errn) ? 0.0 : 1.0, sm) != 0.0) {
            st.finite = false;
            return;
        }
        if (st.it > 1 && st.errn < stop) {
            st.converged = true;
            return;
        }
        if (k + 1 == limit) return;   // the Fock matrix of this iterate is the result
        ++hist;
        const int m = hist < SC_DIIS ? hist : SC_DIIS;
        // new row of the DIIS matrix: <E_i, E_cur>
        {
            double v[SC_DIIS];
            for (int i = 0; i < m; ++i) v[i] = 0.0;
            SC_FOR(t, nn) {
                const double ec = (double)Ec[t];
                for (int i = 0; i < m; ++i) v[i] = fma((double)w.Eh[i * nn + t], ec, v[i]);
            }
            sc_sums(v, m, sm);
            if (tid < m) {
                sm.B[tid][cur] = sm.red[SC_W * SC_DIIS + tid];
                sm.B[cur][tid] = sm.red[SC_W * SC_DIIS + tid];
            }
            __syncthreads();
        }
        // F'_use = sum c_i F'_i (+ level shift (I - P'/2))
        if (m > 1) {
            sc_diis_solve(m, cur, sm);
        } else if (tid == 0) {
            sm.coef[cur] = 1.0;
        }
        __syncthreads();
        SC_FOR(t, nn) {
            T v = T(0);
            if (m > 1) {
                for (int i = 0; i < m; ++i) v = fma((T)sm.coef[i], w.Fh[i * nn + t], v);
            } else {
                v = Fc[t];
            }
            if (a.level_shift != 0.0) {
                const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
                v += (T)a.level_shift * ((mu == nu ? T(1) : T(0)) - T(0.5) * w.Pp[t]);
            }
            w.EA[t] = v;
        }
        sc_bar(sm);
        if constexpr (sizeof(T) == 8) {
            // P' = 2 X, P = X_orth P' X_orth with X_orth = S^-1/2
            if (wait > 0) {
                --wait;
            } else if (sc_purify(n, o, w.EA, w.Pp, w.T1, w.dg, sm)) {
                failed = 0;
                SC_FOR(t, nn) w.Pp[t] *= T(2);
                sc_bar(sm);
                sc_prod(w.dg, n, n, n, T(1), OP_X, w.X, n, false, OP_ANY, w.Pp, n, false, T(0), w.T1, n, false, sm);
                sc_prod(w.dg, n, n, n, T(1), OP_ANY, w.T1, n, false, OP_X, w.X, n, false, T(0), w.P, n, true, sm);
                continue;
            } else {
                wait = 1 << failed;
                if (failed < 5) ++failed;
            }
        }
        if (!sc_eigh<T>(n, o, w.EA, w.Z, w.W, piv, w.dg, sm)) {
            st.finite = false;
            return;
        }
        // P' = 2 Z Z^T, C_o = X Z, P = 2 C_o C_o^T
        sc_prod(w.dg, n, n, o, T(2), OP_ANY, w.Z, o, false, OP_ANY, w.Z, o, true, T(0), w.Pp, n, true, sm);
        sc_prod(w.dg, n, o, n, T(1), OP_X, w.X, n, false, OP_ANY, w.Z, o, false, T(0), w.T2, o, false, sm);
        sc_prod(w.dg, n, n, o, T(2), OP_ANY, w.T2, o, false, OP_ANY, w.T2, o, true, T(0), w.P, n, true, sm);
    }
}

__global__ void __launch_bounds__(SC_T, SC_SLOTS_PER_SM) scc_kernel(ScArgs a) {
    __shared__ ScShared sm;
    const int tid = threadIdx.x;
    const ScSlot sl = sc_slot(a, blockIdx.x / a.csize);
    if (tid == 0) {
        sm.rank = blockIdx.x % a.csize;
        sm.csize = a.csize;
        sm.par = 0;
    }
    __syncthreads();
    sc_bar(sm);   // every CTA of the cluster runs before the first access to its shared memory
    for (int guard = 0; guard < a.n_sys; ++guard) {
        if (tid == 0 && sm.rank == 0) {
            const int nx = atomicAdd(a.next, 1);
            for (int c = 0; c < a.csize; ++c) *(a.csize > 1 ? sc_at(&sm.sys_id, c) : &sm.sys_id) = nx;
        }
        sc_bar(sm);
        const int q = sm.sys_id;
        sc_bar(sm);
        if (q >= a.n_sys) break;
        const int id = a.order[q];
        const tincr_scc_system sy = a.sys[id];
        const int n = sy.n_orb, N = sy.n_atoms, o = sy.n_occ;
        const long long nn = (long long)n * n, NN = (long long)N * N;
        const double erep = sc_setup(a, sy, sl, sm);
        const double *p0 = sl.p0;
        SC_FOR(mu, n) {
            const int A = sm.ao_atom[mu];
            sl.p0[mu] = a.kind_occ[4 * sm.kind[A] + (mu - sm.ao_off[A])];
        }
        ScState st{0, false, 0.0, true};
        ScWork<double> w = sc_work<double>(sl, nn);
        w.S = sl.S; w.H0 = sl.H0; w.X = sl.X; w.Sh = sl.Sh; w.gam = sl.gam; w.glr = sl.glr;
        // X = S^-1/2 and S^1/2 from the eigenpairs of S (scc_routine.rs:172-174)
        SC_FOR(t, nn) w.EA[t] = w.S[t];
        sc_bar(sm);
        bool ok = sc_eigh<double>(n, n, w.EA, w.Z, w.Fh, sl.piv, w.dg, sm);
        if (ok) {
            double bad = 0.0;
            for (int r = tid; r < n; r += SC_T) bad = fmax(bad, sm.w[r] > 0.0 ? 0.0 : 1.0);
            ok = sc_max_cta(bad, sm) == 0.0;
        }
        const double *ps = a.p_start ? a.p_start + sy.mat_off : nullptr;
        auto start_density = [&]() {
            SC_FOR(t, nn) {
                const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
                w.P[t] = ps ? ps[t] : (mu == nu ? p0[mu] : 0.0);
            }
            sc_bar(sm);
        };
        if (ok) {
            SC_FOR(t, nn) {
                const int r = (int)(t % n);
                w.T1[t] = w.Z[t] / sqrt(sm.w[r]);
                w.T2[t] = w.Z[t] * sqrt(sm.w[r]);
            }
            sc_bar(sm);
            gemm_sym<double>(n, n, 1.0, w.T1, n, false, w.Z, n, true, 0.0, w.X, n, sm);
            gemm_sym<double>(n, n, 1.0, w.T2, n, false, w.Z, n, true, 0.0, w.Sh, n, sm);
            if (sc_digits(n, sm)) {
                sc_split(w.S, n, false, n, n, w.dg.S, w.dg.eS, sm);
                sc_split(w.X, n, false, n, n, w.dg.X, w.dg.eX, sm);
            }
            start_density();
        }
        int remaining = a.max_iter, hist = 0;
        if (ok && a.fp32_start) {
            // FP32 phase: its work arrays at the start of the work area, FP32 copies of the inputs
            // after them (the FP64 density in w.P does not overlap either)
            ScWork<float> wf = sc_work<float>(sl, nn);
            float *cp = reinterpret_cast<float *>(sl.work) + (13 + 2 * SC_DIIS) * nn;
            wf.S = cp; wf.H0 = cp + nn; wf.X = cp + 2 * nn; wf.Sh = cp + 3 * nn; wf.gam = cp + 4 * nn;
            wf.glr = wf.gam + NN;
            SC_FOR(t, nn) {
                wf.S[t] = (float)w.S[t];
                wf.H0[t] = (float)w.H0[t];
                wf.X[t] = (float)w.X[t];
                wf.Sh[t] = (float)w.Sh[t];
                wf.P[t] = (float)w.P[t];
            }
            SC_FOR(t, NN) {
                wf.gam[t] = (float)w.gam[t];
                wf.glr[t] = (float)w.glr[t];
            }
            sc_bar(sm);
            const int lim = remaining < SC_FP32_MAX ? remaining : SC_FP32_MAX;
            ScState sf{0, false, 0.0, true};
            sc_iterate<float>(a, sy, wf, sl.piv, p0, lim, fmax(a.tol, SC_FP32_SWITCH), sf, hist, sm);
            if (sf.finite) {
                // continue in FP64 from the density of the FP32 phase's last diagonalisation, with
                // its DIIS history: E' first (FP64 slots beyond every FP32 array), then F' (FP64
                // slots over the FP32 E' and input copies, which are done with)
                SC_FOR(t, nn) w.P[t] = (double)wf.P[t];
                const int m = hist + 1 < SC_DIIS ? hist + 1 : SC_DIIS;
                SC_FOR(t, m * nn) w.Eh[t] = (double)wf.Eh[t];
                sc_bar(sm);
                SC_FOR(t, m * nn) w.Fh[t] = (double)wf.Fh[t];
                sc_bar(sm);
            } else {
                start_density();
                hist = 0;
            }
            st.it = sf.it;
            remaining -= sf.it;
            if (remaining < 1) remaining = 1;
        }
        if (ok) {
            sc_iterate<double>(a, sy, w, sl.piv, p0, remaining, a.tol, st, hist, sm);
            if (!st.finite && a.fp32_start) {
                // the continuation from the FP32 phase failed: max_iter FP64 iterations from the
                // start, with a fresh DIIS history (the iteration count goes on)
                start_density();
                hist = 0;
                st = ScState{st.it, false, 0.0, true};
                sc_iterate<double>(a, sy, w, sl.piv, p0, a.max_iter, a.tol, st, hist, sm);
            }
            ok = st.finite;
        }
        double energy = 0.0;
        if (ok) {
            // orbitals of the last Fock matrix (scc_routine.rs:187-192)
            SC_FOR(t, nn) w.EA[t] = w.Fp[t];
            sc_bar(sm);
            ok = sc_eigh<double>(n, n, w.EA, w.Z, w.Fh, sl.piv, w.dg, sm);
        }
        if (ok) {
            double *C = a.orbs + sy.mat_off;
            gemm<double>(n, n, n, 1.0, w.X, n, false, w.Z, n, false, 0.0, C, n, sm);
            gemm_sym<double>(n, o, 2.0, C, n, false, C, n, true, 0.0, w.P, n, sm);
            sc_charges<double>(n, N, w.P, w.S, w.gam, p0, sm);
            // E = sum P o H0 + 1/2 dq gamma dq [- 1/8 (sum (S dP S) o dP o g_lr + sum (S dP) o (dP S) o g_lr)]
            double e1 = 0.0;
            SC_FOR(t, nn) e1 = fma(w.P[t], w.H0[t], e1);
            double e2 = 0.0;
            SC_FOR(A, N) e2 += 0.5 * sm.dq[A] * sm.esp[A];
            double e3 = 0.0;
            if (a.lc) {
                double *dP = w.W;
                SC_FOR(t, nn) {
                    const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
                    dP[t] = w.P[t] - (mu == nu ? p0[mu] : 0.0);
                }
                sc_bar(sm);
                gemm<double>(n, n, n, 1.0, w.S, n, false, dP, n, false, 0.0, w.T1, n, sm);
                gemm_sym<double>(n, n, 1.0, w.T1, n, false, w.S, n, false, 0.0, w.T2, n, sm);
                SC_FOR(t, nn) {
                    const int mu = (int)(t / n), nu = (int)(t - (long long)mu * n);
                    const double g = w.glr[(long long)sm.ao_atom[mu] * N + sm.ao_atom[nu]];
                    e3 += g * (w.T2[t] * dP[t] + w.T1[t] * w.T1[(long long)nu * n + mu]);
                }
                e3 *= -0.125;
            }
            energy = sc_sum(e1 + e2 + e3, sm) + erep;
            SC_FOR(r, n) a.orbe[sy.orb_off + r] = sm.w[r];
            SC_FOR(A, N) a.dq[sy.atom_off + A] = sm.dq[A];
            SC_FOR(t, nn) {
                if (a.p) a.p[sy.mat_off + t] = w.P[t];
                if (a.s_out) a.s_out[sy.mat_off + t] = w.S[t];
                if (a.h0_out) a.h0_out[sy.mat_off + t] = w.H0[t];
                if (a.hcx) a.hcx[sy.mat_off + t] = w.F[t];
            }
        }
        if (tid == 0 && sm.rank == 0) {
            a.iterations[id] = st.it;
            a.converged[id] = (ok && st.converged) ? 1 : 0;
            a.residual[id] = ok ? st.errn : NAN;
            a.energy[id] = ok ? energy : NAN;
            a.status[id] = ok ? TINCR_OK : TINCR_NONFINITE;
        }
        sc_bar(sm);
    }
}

// CTAs per system, one for the whole batch: the largest power of two that keeps it within `fill` CTAs per SM.
// What the size of its systems allows is measured by their mean weighted with the cube, the work of an
// iteration (a few large systems decide, a few large ones among thousands of small ones do not).  Below 16
// orbitals a second CTA only adds barriers; below SC_SMALL the systems of a batch converge alike, so more
// than what runs at once is a second wave, while the larger ones (dimers) differ by hundreds of iterations
// and the last ones are worth the CTAs; up to 112 orbitals short of a full second wave (152 pentacenes without
// LC on 4 CTAs 78.8 ms, on 2 49.6; from the FP32 start 73.7 and 43.9, 68.4 with one CTA and the eigensolver;
// 152 stacked naphthalene dimers 542 and 582).  Clusters of 16 fit on a GPC a few at a time, so small systems take
// them up to four.  Kernel time (ms, LC, to 1e-10) with one CTA and the eigensolver in every iteration / two
// CTAs and more, SC_FILL CTAs per SM for all / this rule:
//     304 systems of 6 orbitals  1.74 / 3.89 / 1.51     304 of 30 orbitals  11.5 / 16.5 /  8.1
//      64 of 6                   1.60 / 3.73 / 1.26     152 of 30           10.3 / 15.5 /  6.3
//     304 of 12                  2.79 / 4.75 / 1.96     152 of 48           23.0 / 32.3 / 14.3
//     304 of 24                  6.83 / 8.55 / 5.03     152 of 66           56.9 / 48.5 / 28.6
int sc_ctas_per_system(int n_sys, const tincr_scc_system *sys, int n_sm) {
    double w3 = 0.0, w4 = 0.0;
    for (int i = 0; i < n_sys; ++i) {
        const double n = sys[i].n_orb;
        w3 += n * n * n;
        w4 += n * n * n * n;
    }
    const double size = w4 / w3;
    const bool small = size < SC_SMALL;
    const double fill = size < 32.0 ? 1.0 : small ? 2.0 : size < 112.0 ? 3.5 : SC_FILL;
    const int most = size < 16.0 ? 1 : size < 32.0 ? 4 : small && n_sys > 4 ? 8 : SC_CMAX;
    int csize = small ? 1 : 2;
    while (csize < most && 2.0 * csize * n_sys <= fill * n_sm) csize *= 2;
    return csize;
}

}  // namespace

int Ctx::scc_batch(int n_sys, const tincr_scc_system *sys, const int *kinds, const double *xyz,
                   const double *kind_energy, const tincr_scc_inputs *given, const double *p_start, double r_lr,
                   int flags, double tol, int max_iter,
                   double level_shift, double *orbe, double *orbs, double *p_out, double *dq, double *energy,
                   double *s_out, double *h0_out, double *hcx_out, int *iterations, int *converged,
                   double *residual) {
    if (!params_ready) fail(TINCR_BAD_ARG, "scc_batch: tincr_set_parameters first");
    if (n_sys < 1 || !sys || !kinds || !xyz || !kind_energy || !orbe || !orbs || !energy || !iterations ||
        !converged || !residual)
        fail(TINCR_BAD_ARG, "scc_batch: bad arguments");
    if (!(tol > 0.0) || max_iter < 1 || !std::isfinite(level_shift) || level_shift < 0.0)
        fail(TINCR_BAD_ARG, "scc_batch: tol > 0, max_iter >= 1, level_shift >= 0");
    const bool lc = (flags & TINCR_SCC_LC) != 0;
    if (lc && !(r_lr > 0.0)) fail(TINCR_BAD_ARG, "scc_batch: LC needs r_lr > 0");
    if (flags & ~(TINCR_SCC_LC | TINCR_SCC_SK_EXTRAPOLATE | TINCR_SCC_FP32_START))
        fail(TINCR_BAD_ARG, "scc_batch: unknown flags");
    long long n_at_tot = 0, n_orb_tot = 0, n_mat_tot = 0, n_pair_tot = 0;
    int nmax = 0, Nmax = 0;
    for (int i = 0; i < n_sys; ++i) {
        const tincr_scc_system &s = sys[i];
        if (s.n_atoms < 1 || s.n_atoms > SC_NMAX || s.n_orb < 2 || s.n_orb > SC_NMAX || s.n_occ < 1 ||
            s.n_occ > s.n_orb || s.atom_off < 0 || s.orb_off < 0 || s.mat_off < 0 || s.pair_off < 0)
            fail(TINCR_BAD_ARG, "scc_batch: system " + std::to_string(i) + ": sizes or offsets out of range "
                                "(2 <= n_orb <= 256, 1 <= n_atoms <= 256, 1 <= n_occ <= n_orb)");
        int no = 0;
        for (int A = 0; A < s.n_atoms; ++A) {
            const int k = kinds[s.atom_off + A];
            if (k < 0 || k >= n_kinds) fail(TINCR_BAD_ARG, "scc_batch: atom kind out of range");
            no += h_kind_norb[k];
        }
        if (no != s.n_orb) fail(TINCR_BAD_ARG, "scc_batch: n_orb does not match the atoms' orbitals");
        n_at_tot = std::max(n_at_tot, s.atom_off + s.n_atoms);
        n_orb_tot = std::max(n_orb_tot, s.orb_off + s.n_orb);
        n_mat_tot = std::max(n_mat_tot, s.mat_off + (long long)s.n_orb * s.n_orb);
        n_pair_tot = std::max(n_pair_tot, s.pair_off + (long long)s.n_atoms * s.n_atoms);
        nmax = std::max(nmax, s.n_orb);
        Nmax = std::max(Nmax, s.n_atoms);
    }
    for (long long i = 0; i < 3 * n_at_tot; ++i)
        if (!std::isfinite(xyz[i])) fail(TINCR_NONFINITE, "scc_batch: non-finite coordinates");
    for (int i = 0; i < 4 * n_kinds; ++i)
        if (!std::isfinite(kind_energy[i])) fail(TINCR_NONFINITE, "scc_batch: non-finite orbital energies");
    auto finite = [](const double *x, long long len, const char *what) {
        if (x)
            for (long long i = 0; i < len; ++i)
                if (!std::isfinite(x[i])) fail(TINCR_NONFINITE, std::string("scc_batch: non-finite ") + what);
    };
    const tincr_scc_inputs none{nullptr, nullptr, nullptr, nullptr};
    const tincr_scc_inputs &gv = given ? *given : none;
    finite(p_start, n_mat_tot, "starting density");
    finite(gv.s, n_mat_tot, "S");
    finite(gv.h0, n_mat_tot, "H0");
    finite(gv.gamma, n_pair_tot, "gamma");
    finite(gv.gamma_lr, lc ? n_pair_tot : 0, "gamma_lr");
    // largest systems first
    std::vector<int> order(n_sys);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return sys[x].n_orb > sys[y].n_orb; });
    // device copies
    DevBuf<tincr_scc_system> d_sys(n_sys);
    DevBuf<int> d_order(n_sys), d_kind(n_at_tot), d_ints(4 * (size_t)n_sys + 1);
    DevBuf<double> d_xyz3(3 * n_at_tot), d_ke(4 * (size_t)n_kinds), d_occ(4 * (size_t)n_kinds);
    DevBuf<double> d_ps(p_start ? n_mat_tot : 0), d_orbe(n_orb_tot), d_orbs(n_mat_tot), d_dq(n_at_tot);
    DevBuf<double> d_p(p_out ? n_mat_tot : 0), d_s(s_out ? n_mat_tot : 0), d_h0(h0_out ? n_mat_tot : 0);
    DevBuf<double> d_hcx(hcx_out ? n_mat_tot : 0), d_sc(2 * (size_t)n_sys);
    DevBuf<double> d_sin(gv.s ? n_mat_tot : 0), d_h0in(gv.h0 ? n_mat_tot : 0);
    DevBuf<double> d_gin(gv.gamma ? n_pair_tot : 0), d_glrin(gv.gamma_lr && lc ? n_pair_tot : 0);
    auto up = [&](void *dst, const void *src, size_t bytes) {
        TINCR_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream));
    };
    up(d_sys.p, sys, sizeof(tincr_scc_system) * n_sys);
    up(d_order.p, order.data(), sizeof(int) * n_sys);
    up(d_kind.p, kinds, sizeof(int) * n_at_tot);
    up(d_xyz3.p, xyz, sizeof(double) * 3 * n_at_tot);
    up(d_ke.p, kind_energy, sizeof(double) * 4 * n_kinds);
    up(d_occ.p, h_kind_occ.data(), sizeof(double) * 4 * n_kinds);
    if (p_start) up(d_ps.p, p_start, sizeof(double) * n_mat_tot);
    if (gv.s) up(d_sin.p, gv.s, sizeof(double) * n_mat_tot);
    if (gv.h0) up(d_h0in.p, gv.h0, sizeof(double) * n_mat_tot);
    if (gv.gamma) up(d_gin.p, gv.gamma, sizeof(double) * n_pair_tot);
    if (gv.gamma_lr && lc) up(d_glrin.p, gv.gamma_lr, sizeof(double) * n_pair_tot);
    TINCR_CUDA(cudaMemsetAsync(d_ints.p, 0, sizeof(int) * (4 * (size_t)n_sys + 1), stream));
    // slots
    const long long nn_max = (long long)nmax * nmax, at2_max = (long long)Nmax * Nmax, npad = (nmax + 31) / 32 * 32;
    const long long slot_bytes =
        (sc_slot_doubles(nn_max, at2_max, npad) * (long long)sizeof(double) + nn_max + 255) / 256 * 256 + sc_digit_bytes(npad);
    const int csize = sc_ctas_per_system(n_sys, sys, n_sm);
    const int n_slots = std::min(n_sys, SC_SLOTS_PER_SM * n_sm / csize);
    scc_ws.reserve((size_t)(slot_bytes * n_slots));
    ScArgs a{};
    a.n_sys = n_sys;
    a.sys = d_sys.p;
    a.order = d_order.p;
    a.kind = d_kind.p;
    a.xyz = d_xyz3.p;
    a.p_start = p_start ? d_ps.p : nullptr;
    a.s_in = gv.s ? d_sin.p : nullptr;
    a.h0_in = gv.h0 ? d_h0in.p : nullptr;
    a.gam_in = gv.gamma ? d_gin.p : nullptr;
    a.glr_in = gv.gamma_lr && lc ? d_glrin.p : nullptr;
    a.n_kinds = n_kinds;
    a.n_knots = n_knots;
    a.sk_extrapolate = (flags & TINCR_SCC_SK_EXTRAPOLATE) ? 1 : 0;
    a.kind_z = d_kind_z.p;
    a.kind_norb = d_kind_norb.p;
    a.kind_l = d_kind_l.p;
    a.kind_m = d_kind_m.p;
    a.kind_occ = d_occ.p;
    a.kind_energy = d_ke.p;
    a.sigma = d_sigma.p;
    a.knots = d_knots.p;
    a.coef = d_coef.p;
    a.rep_ntmax = rep_ntmax;
    a.rep_nt = rep_ntmax > 0 ? d_rep_nt.p : nullptr;
    a.rep_knots = d_rep_knots.p;
    a.rep_coef = d_rep_coef.p;
    a.rep_dmax = d_rep_dmax.p;
    a.lc = lc ? 1 : 0;
    a.r_lr = lc ? r_lr : 0.0;
    a.tol = tol;
    a.level_shift = level_shift;
    a.max_iter = max_iter;
    a.fp32_start = (flags & TINCR_SCC_FP32_START) ? 1 : 0;
    a.orbe = d_orbe.p;
    a.orbs = d_orbs.p;
    a.p = p_out ? d_p.p : nullptr;
    a.dq = d_dq.p;
    a.energy = d_sc.p;
    a.residual = d_sc.p + n_sys;
    a.s_out = s_out ? d_s.p : nullptr;
    a.h0_out = h0_out ? d_h0.p : nullptr;
    a.hcx = hcx_out ? d_hcx.p : nullptr;
    a.iterations = d_ints.p;
    a.converged = d_ints.p + n_sys;
    a.status = d_ints.p + 2 * n_sys;
    a.next = d_ints.p + 4 * n_sys;
    a.ws = scc_ws.p;
    a.slot_bytes = slot_bytes;
    a.nn_max = nn_max;
    a.at2_max = at2_max;
    a.npad = npad;
    TINCR_CUDA(cudaEventRecord(ev0, stream));
    g_launches = 0;
    a.csize = csize;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(n_slots * csize));
    cfg.blockDim = dim3(SC_T);
    cfg.stream = stream;
    cudaLaunchAttribute cl[1];
    cl[0].id = cudaLaunchAttributeClusterDimension;
    cl[0].val.clusterDim.x = (unsigned)csize;
    cl[0].val.clusterDim.y = cl[0].val.clusterDim.z = 1;
    cfg.attrs = cl;
    cfg.numAttrs = 1;
    if (csize > 8) TINCR_CUDA(cudaFuncSetAttribute(scc_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    TINCR_CUDA(cudaLaunchKernelEx(&cfg, scc_kernel, a));
    count_launch(stream, "scc_kernel");
    check_launch("scc_kernel");
    TINCR_CUDA(cudaEventRecord(ev1, stream));
    auto down = [&](void *dst, const void *src, size_t bytes) {
        TINCR_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream));
    };
    std::vector<int> ints(3 * (size_t)n_sys);
    std::vector<double> sc(2 * (size_t)n_sys);
    down(ints.data(), d_ints.p, sizeof(int) * 3 * n_sys);
    down(sc.data(), d_sc.p, sizeof(double) * 2 * n_sys);
    down(orbe, d_orbe.p, sizeof(double) * n_orb_tot);
    down(orbs, d_orbs.p, sizeof(double) * n_mat_tot);
    if (dq) down(dq, d_dq.p, sizeof(double) * n_at_tot);
    if (p_out) down(p_out, d_p.p, sizeof(double) * n_mat_tot);
    if (s_out) down(s_out, d_s.p, sizeof(double) * n_mat_tot);
    if (h0_out) down(h0_out, d_h0.p, sizeof(double) * n_mat_tot);
    if (hcx_out) down(hcx_out, d_hcx.p, sizeof(double) * n_mat_tot);
    sync();
    float ms = 0.f;
    TINCR_CUDA(cudaEventElapsedTime(&ms, ev0, ev1));
    last_ms = ms;
    last_launches = g_launches;
    int rc = TINCR_OK;
    for (int i = 0; i < n_sys; ++i) {
        iterations[i] = ints[i];
        converged[i] = ints[n_sys + i];
        energy[i] = sc[i];
        residual[i] = sc[n_sys + i];
        if (ints[2 * n_sys + i] == TINCR_NONFINITE) rc = TINCR_NONFINITE;
        else if (!ints[n_sys + i] && rc == TINCR_OK) rc = TINCR_NOT_CONVERGED;
    }
    if (rc == TINCR_NONFINITE) err = "scc_batch: non-finite value in an SCC iteration (see the per-system residual)";
    else if (rc == TINCR_NOT_CONVERGED) err = "scc_batch: some systems did not converge (see converged[])";
    return rc;
}

}  // namespace tincr
