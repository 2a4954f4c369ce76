// Batched FP64 GEMM with fused epilogues (SIMT, shared-memory tiled).
//
// C_b(m, n) = epi( sum_k op(A_b)(m, k) * op(B_b)(k, n) ) for b in [0, batch), row-major storage:
//   op(A)(m, k) = TA ? A[k*lda + m] : A[m*lda + k]
//   op(B)(k, n) = TB ? B[n*ldb + k] : B[k*ldb + n]
// 16- or 32-deep k slices are staged through shared memory with a register prefetch of the next
// slice.  Split-K over blockIdx.z (for the tall-skinny subspace products, whose K is the full
// singles space) hands partial sums to an accumulating epilogue.
//
// GB300's FP64 rate (about 2 DFMA per SM clock, one warp instruction per 64 clocks and SM
// sub-partition) makes every FP64 contraction of this path DFMA-bound: a T x T tile costs T T K / 2
// clocks of its SM whatever its shared-memory traffic, padding included, and a product of a small
// system has few tiles.  So the tile is the one of 64x64, 32x32, 16x16 (256 threads) and 8x16 (128
// threads, the four sub-partitions) whose largest per-SM share of padded outputs is least
// (f64_tile_for).  Every output is one fma chain over ascending k in every tile, so the choice does
// not change a bit.  Measured against 64x64 alone: S0 + S1 gradient of decacene (n = 192) 79.8 ->
// 10.2 ms, one A.X product of naphthalene (n = 48) 334 -> 79 us per call, 20 products of (H2O)128
// kept on the tiles (n = 768, 64x64 still chosen for most of it; large work runs on digits, contract_digits.cu)
// 55.6 -> 54.4 ms.  Even 16x16 with one output per thread stays pipe-bound: two shared-memory wavefronts and
// 2 bytes of operands per 16 clocks.
#pragma once

#include "common.cuh"

namespace tincr {

constexpr int GB_M = 64, GB_N = 64, GB_K = 16, GB_T = 256;

// Plain store: C = alpha * acc + beta * C
struct EpiStore {
    double *C;
    long long sC;
    int ldc;
    double alpha, beta;
    __device__ __forceinline__ void operator()(int b, int m, int n, double acc) const {
        double *p = C + b * sC + (long long)m * ldc + n;
        *p = (beta == 0.0) ? alpha * acc : alpha * acc + beta * (*p);
    }
};

// Accumulate (split-K partial sums): C += alpha * acc
struct EpiAtomicAdd {
    double *C;
    long long sC;
    int ldc;
    double alpha;
    __device__ __forceinline__ void operator()(int b, int m, int n, double acc) const {
        atomicAdd(C + b * sC + (long long)m * ldc + n, alpha * acc);
    }
};

// Tile of TM x TN outputs by TY x TX threads, KS deep slices.
template <int TY, int TX, int R, int KS_>
struct F64Tile {
    static constexpr int M = TY * R, N = TX * R, KS = KS_, T = TX * TY, X = TX, Y = TY, O = R;
};
using F64T64 = F64Tile<16, 16, 4, 16>;
using F64T32 = F64Tile<16, 16, 2, 16>;
using F64T16 = F64Tile<16, 16, 1, 32>;
using F64T8 = F64Tile<8, 16, 1, 32>;

// One output tile over k in [kbeg, kend): acc[i][j] holds C(m0 + ty + Y i, n0 + tx + X j) for thread
// (tx, ty) = (tid % X, tid / X).  All W::T threads take part.
template <class W, bool TA, bool TB>
__device__ __forceinline__ void f64_tile(int M, int N, int kbeg, int kend, const double *__restrict__ A, int lda,
                                         const double *__restrict__ B, int ldb, int m0, int n0,
                                         double (&As)[W::KS][W::M + 1], double (&Bs)[W::KS][W::N + 1],
                                         double (&acc)[W::O][W::O]) {
    constexpr int EA = W::M * W::KS / W::T, EB = W::N * W::KS / W::T;
    const int tid = threadIdx.x, tx = tid % W::X, ty = tid / W::X;
#pragma unroll
    for (int i = 0; i < W::O; ++i)
#pragma unroll
        for (int j = 0; j < W::O; ++j) acc[i][j] = 0.0;
    double ra[EA], rb[EB];
    // consecutive threads read consecutive addresses of either layout
    auto load = [&](int k0) {
#pragma unroll
        for (int e = 0; e < EA; ++e) {
            const int idx = e * W::T + tid;
            const int m = m0 + (TA ? idx % W::M : idx / W::KS), k = k0 + (TA ? idx / W::M : idx % W::KS);
            ra[e] = (m < M && k < kend) ? (TA ? A[(long long)k * lda + m] : A[(long long)m * lda + k]) : 0.0;
        }
#pragma unroll
        for (int e = 0; e < EB; ++e) {
            const int idx = e * W::T + tid;
            const int n = n0 + (TB ? idx / W::KS : idx % W::N), k = k0 + (TB ? idx % W::KS : idx / W::N);
            rb[e] = (n < N && k < kend) ? (TB ? B[(long long)n * ldb + k] : B[(long long)k * ldb + n]) : 0.0;
        }
    };
    auto store = [&]() {
#pragma unroll
        for (int e = 0; e < EA; ++e) {
            const int idx = e * W::T + tid;
            As[TA ? idx / W::M : idx % W::KS][TA ? idx % W::M : idx / W::KS] = ra[e];
        }
#pragma unroll
        for (int e = 0; e < EB; ++e) {
            const int idx = e * W::T + tid;
            Bs[TB ? idx % W::KS : idx / W::N][TB ? idx / W::KS : idx % W::N] = rb[e];
        }
    };
    if (kbeg < kend) {
        load(kbeg);
        for (int k0 = kbeg; k0 < kend; k0 += W::KS) {
            __syncthreads();
            store();
            __syncthreads();
            if (k0 + W::KS < kend) load(k0 + W::KS);
            // the last slice stops at kend: a k past it is an FP64 instruction that adds zero
            const int kn = kend - k0 < W::KS ? kend - k0 : W::KS;
            auto step = [&](int kk) {
                double a[W::O], b[W::O];
#pragma unroll
                for (int i = 0; i < W::O; ++i) a[i] = As[kk][ty + W::Y * i];
#pragma unroll
                for (int j = 0; j < W::O; ++j) b[j] = Bs[kk][tx + W::X * j];
#pragma unroll
                for (int i = 0; i < W::O; ++i)
#pragma unroll
                    for (int j = 0; j < W::O; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            };
            if (kn == W::KS) {
#pragma unroll
                for (int kk = 0; kk < W::KS; ++kk) step(kk);
            } else {
                for (int kk = 0; kk < kn; ++kk) step(kk);
            }
        }
    }
}

template <class W, bool TA, bool TB, class Epi>
__global__ void __launch_bounds__(W::T)
gemm_f64_kernel(int M, int N, int K, int k_chunk, int splitk, const double *__restrict__ A, int lda,
                long long sA, const double *__restrict__ B, int ldb, long long sB, Epi epi) {
    __shared__ double As[W::KS][W::M + 1];
    __shared__ double Bs[W::KS][W::N + 1];
    const int tx = threadIdx.x % W::X, ty = threadIdx.x / W::X;
    const int zb = blockIdx.z / splitk, zk = blockIdx.z % splitk;
    const int m0 = blockIdx.y * W::M, n0 = blockIdx.x * W::N;
    const int kbeg = zk * k_chunk;
    const int kend = min(K, kbeg + k_chunk);
    double acc[W::O][W::O];
    f64_tile<W, TA, TB>(M, N, kbeg, kend, A + zb * sA, lda, B + zb * sB, ldb, m0, n0, As, Bs, acc);
#pragma unroll
    for (int i = 0; i < W::O; ++i) {
        const int m = m0 + ty + W::Y * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < W::O; ++j) {
            const int n = n0 + tx + W::X * j;
            if (n < N) epi(zb, m, n, acc[i][j]);
        }
    }
}

// The tile edge (64, 32, 16, or 8 for 8 x 16) with the smallest largest per-SM share of padded
// outputs, z products of M x N on n_sm SMs.  A smaller tile has to win by 1/16: its loads per
// output are twice those of the next larger one.
inline int f64_tile_for(int M, int N, long long z, int n_sm) {
    const int tm[4] = {64, 32, 16, 8}, tn[4] = {64, 32, 16, 16};
    int best = 0;
    long long cost = 0;
    for (int i = 0; i < 4; ++i) {
        const long long tiles = (long long)ceil_div(M, tm[i]) * ceil_div(N, tn[i]) * z;
        const long long c = (tiles + n_sm - 1) / n_sm * tm[i] * tn[i];
        if (i == 0 || c * 16 < cost * 15) {
            best = i;
            cost = c;
        }
    }
    return tm[best];
}

// Launch helper.  splitk > 1 requires an accumulating epilogue.
template <class W, bool TA, bool TB, class Epi>
void gemm_f64_launch(cudaStream_t st, int M, int N, int K, int k_chunk, int splitk, const double *A, int lda,
                     long long sA, const double *B, int ldb, long long sB, int batch, Epi epi) {
    dim3 grid(ceil_div(N, W::N), ceil_div(M, W::M), batch * splitk);
    gemm_f64_kernel<W, TA, TB, Epi><<<grid, W::T, 0, st>>>(M, N, K, k_chunk, splitk, A, lda, sA, B, ldb, sB, epi);
    count_launch(st, "gemm_f64");
    check_launch("gemm_f64");
}

template <bool TA, bool TB, class Epi>
void gemm_f64(cudaStream_t st, int n_sm, int M, int N, int K, const double *A, int lda, long long sA,
              const double *B, int ldb, long long sB, int batch, Epi epi, int splitk = 1) {
    if (M <= 0 || N <= 0 || batch <= 0) return;
    if (splitk < 1) splitk = 1;
    int k_chunk = (K + splitk - 1) / splitk;
    k_chunk = ((k_chunk + GB_K - 1) / GB_K) * GB_K;
    if (k_chunk <= 0) k_chunk = GB_K;
    splitk = (K + k_chunk - 1) / k_chunk;
    if (splitk < 1) splitk = 1;
    auto go = [&](auto w) {
        gemm_f64_launch<decltype(w), TA, TB>(st, M, N, K, k_chunk, splitk, A, lda, sA, B, ldb, sB, batch, epi);
    };
    switch (f64_tile_for(M, N, (long long)batch * splitk, n_sm)) {
        case 64: go(F64T64{}); break;
        case 32: go(F64T32{}); break;
        case 16: go(F64T16{}); break;
        default: go(F64T8{}); break;
    }
}

// Split-K factor that fills the GPU for a small M x N output with a long K.
inline int pick_splitk(int M, int N, int K, int batch, int n_sm) {
    long long tiles = (long long)ceil_div(M, GB_M) * ceil_div(N, GB_N) * batch;
    long long want = 4LL * n_sm;
    if (tiles >= want) return 1;
    long long s = (want + tiles - 1) / tiles;
    long long max_s = (K + 255) / 256;   // keep at least 256 k per split
    if (s > max_s) s = max_s;
    return s < 1 ? 1 : int(s);
}

}  // namespace tincr
