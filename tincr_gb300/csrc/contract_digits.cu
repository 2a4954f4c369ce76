// The FP64 AO-direct contraction (Ctx::ao_contract) as FP64-accurate digit GEMMs on the tensor cores.
//
// GB300 issues 2 FP64 FMAs per SM and clock (about 0.6 T FMA/s), so the four products of a
// contraction, 8 nov + 16 n^2 v flops per vector, are bound by the FP64 pipe by a factor of tens over
// everything else.  Here each is a digit GEMM (digits.cuh: eight digits per operand value below its
// row's power-of-two bound, exact integer sums, one rounding per result):
//   H   [2n x |S|]  = [C_R;SC_R] V                     A = V^T,        B = [C_R;SC_R]
//   F   [2n x 2n]   = ax gamma_lr o (H [C_S;SC_S]^T)   A = [C_S;SC_S], B = H       (+ Coulomb diagonals)
//   G^T [|Q| x 2n]  = (F [SC_Q;C_Q])^T                 A = F,          B = [SC_Q;C_Q]^T
//   out [|P| x |Q|] = [SC_P;C_P]^T G (+ omega o X)     A = G^T,        B = [SC_P;C_P]^T
// Every GEMM computes C(col, row) for row = an A row (one lane each) and col = a B row and stores it
// at [col][row]: the lanes of a warp store 32 consecutive doubles, and the result is laid out as the
// K-major rows that the next product reads.  Its epilogue also takes the row maxima that the next
// split needs (redux over the warp, one 32-bit atomicMax on the high words per column), so a split
// is one pass: FP64 in, digit planes out.  The digits of the orbital blocks are cut once per system.
//
// The digits are those of fixed8.cuh.  (Digits of 7 bits with x's sign, which truncate towards zero, gave
// A.X errors 3 to 6 times those of the FP64 FMAs.)
//
// Precision.  A value is held to 2^-62 of its row's largest, so the error of a result is relative to the
// largest values of two rows and not to each of its terms.  Error of A.X in the norm against quad precision,
// digits / FP64 tiles: naphthalene .. decacene, (H2O)16, (H2O)40, C20H22 7.1e-17 .. 8.5e-17 / 7.3e-17 ..
// 1.0e-16; (H2O)24 and two naphthalenes 22 to 1000 bohr apart, each with a random, a unit, a steep and a graded
// vector, 2.1e-17 .. 1.2e-16 / 2.1e-17 .. 1.8e-16.  The components are as good as the tiles' (medians 5e-17 to
// 2e-15) but for those 2^-50 and more below their rows' largest: of a unit vector on one of two far fragments,
// components of 1e-20 keep eight digits or fewer (the tiles: fourteen).  TINCR_GB300_CONTRACTION=fp64 keeps
// the tiles.
//
// What bounds it: 36 digit products per FMA on the tensor cores (2.3 TFLOP of bf16 at 20 vectors of
// (H2O)128, 1.2 ms at the measured GEMM rate) and the F planes (16 bytes per element, written and read
// once).  20 products of (H2O)128 (n = 768, 32 G FMA) take 2.5 ms on the device, 52.6 ms on FP64 tiles
// (0.6 T FMA/s, the FP64 pipe).  The tiles stay the better path for small work (digits_pay).
#include <algorithm>

#include "digits.cuh"
#include "fixed8.cuh"
#include "kernels.cuh"
#include "ops.cuh"
#include "tda.cuh"

namespace tincr {

namespace {

// Source of a digit operand: row r, element k of product b at p[b * sb + r * rs + k * ks] (one of
// rs, ks is 1), R rows of K elements.
struct CdSrc {
    const double *p;
    long long sb, rs, ks;
    int R, K;
};

// 32 rows x 64 k of a source per CTA of 256 threads, thread (row t / 8, k 8 (t % 8) ..) of it; reads
// are coalesced along the contiguous axis (rows contiguous: through shared memory)
__device__ __forceinline__ void cd_load(const CdSrc &s, int b, int r0, int k0, double (&x)[8], double (*st)[33]) {
    const int t = threadIdx.x, r = r0 + (t >> 3), k = k0 + 8 * (t & 7);
    const double *p = s.p + (long long)b * s.sb;
    if (s.ks == 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = (r < s.R && k + j < s.K) ? p[(long long)r * s.rs + k + j] : 0.0;
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int kk = (t >> 5) + 8 * j, rr = t & 31;
        st[kk][rr] = (r0 + rr < s.R && k0 + kk < s.K) ? p[(long long)(r0 + rr) * s.rs + (long long)(k0 + kk) * s.ks] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = st[8 * (t & 7) + j][t >> 3];
}

// mx[b * rows_pad + r] = largest high word of row r; grid (k blocks, row blocks, products), mx zeroed
__global__ void __launch_bounds__(256) cd_max_kernel(CdSrc s, int rows_pad, unsigned *mx) {
    __shared__ double st[64][33];
    double x[8];
    cd_load(s, blockIdx.z, blockIdx.y * 32, blockIdx.x * 64, x, st);
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) m = max(m, cd_hi_any(x[j]));
    for (int o = 4; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int r = blockIdx.y * 32 + (threadIdx.x >> 3);
    if ((threadIdx.x & 7) == 0 && m) atomicMax(mx + (long long)blockIdx.z * rows_pad + r, m);
}

// digit planes of a source (zeros in the padding rows and k) and the bound exponents of its rows
__global__ void __launch_bounds__(256) cd_split_kernel(CdSrc s, int rows_pad, const unsigned *__restrict__ mx,
                                                       DgOperand op, int *E) {
    __shared__ double st[64][33];
    double x[8];
    const int b = blockIdx.z, r = blockIdx.y * 32 + (threadIdx.x >> 3), k = blockIdx.x * 64 + 8 * (threadIdx.x & 7);
    cd_load(s, b, blockIdx.y * 32, blockIdx.x * 64, x, st);
    const long long row = (long long)b * rows_pad + r;
    const int e = r < s.R ? cd_bound(mx[row]) : 0;
    if (blockIdx.x == 0 && (threadIdx.x & 7) == 0) E[row] = e;
    unsigned long long y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = cd_fixed<true>(e == CD_POISON ? 0.0 : x[j], e);
#pragma unroll
    for (int p = 0; p < DG_PLANES; ++p) {
        unsigned w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = cd_pair(y[2 * j], y[2 * j + 1], p);
        *reinterpret_cast<uint4 *>(op.p + dg_off(op, p, row, k)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// sum over k of A(row, k) B(col, k) in FP64, k ascending: the results of a row without digits, which holds an
// overflow of an earlier product
__device__ __noinline__ double cd_direct(const CdSrc &A, const CdSrc &B, int b, int row, int col) {
    const double *p = A.p + (long long)b * A.sb + (long long)row * A.rs;
    const double *q = B.p + (long long)b * B.sb + (long long)col * B.rs;
    double v = 0.0;
    for (int k = 0; k < A.K; ++k) v = fma(p[(long long)k * A.ks], q[(long long)k * B.ks], v);
    return v;
}

// Values of one thread's 16 results: A row `row` (bound Ea), B rows col0 .. col0 + 15 (bounds Eb)
struct CdScale {
    const int *Ea, *Eb;   // per product: ea_b, eb_b entries further (0: shared)
    int ea_b, eb_b;
    CdSrc A, B;           // what the digits were cut from
    __device__ __forceinline__ int row(int b, int r) const { return Ea[(long long)b * ea_b + r]; }
    __device__ __forceinline__ double value(int b, int row, int ea, int col, long long H, long long L) const {
        const int eb = Eb[(long long)b * eb_b + col];
        const int e = ea + eb - 68;   // beyond every sum of two bounds where one row has no digits
        return __longlong_as_double((long long)cd_value_bits(H, L, e, [&](unsigned long long m, int ex, unsigned long long s) {
            if (e > CD_POISON / 2) return (unsigned long long)__double_as_longlong(cd_direct(A, B, b, row, col));
            return cd_extreme(m, ex, s);
        }));
    }
};

// C_b[col * ld + row] = v, and the largest |v| of each col into mx (per product mx_b entries further)
struct CdEpiStore {
    static constexpr int BITS = 8;
    CdScale sc;
    double *C;
    long long sC;
    int ld, M, N;
    unsigned *mx;
    int mx_b;
    __device__ __forceinline__ void operator()(int b, int row, int col0, const long long (&H)[16],
                                               const long long (&L)[16]) const {
        const int ea = row < M ? sc.row(b, row) : 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int col = col0 + j;
            if (col >= N) break;   // uniform over the warp
            double v = 0.0;
            if (row < M) {
                v = sc.value(b, row, ea, col, H[j], L[j]);
                C[(long long)b * sC + (long long)col * ld + row] = v;
            }
            const unsigned m = __reduce_max_sync(0xffffffffu, cd_hi_any(v));
            if ((threadIdx.x & 31) == 0 && m) atomicMax(mx + (long long)b * mx_b + col, m);
        }
    }
};

// F_b[r = col][c = row] = ax gamma_lr[r][c] M(r, c), the diagonals of M's off-diagonal blocks for the
// Coulomb term (M3 = block (0,1), M2 = block (1,0)), and the row maxima of F
struct CdEpiF {
    static constexpr int BITS = 8;
    CdScale sc;
    double *F;
    long long sF;
    int ld, n;
    const double *G;   // n x n
    double ax;
    double *d3, *d2;   // [product][n]
    unsigned *mx;
    int mx_b;
    __device__ __forceinline__ void operator()(int b, int row, int col0, const long long (&H)[16],
                                               const long long (&L)[16]) const {
        const int n2 = 2 * n, ea = row < n2 ? sc.row(b, row) : 0, cc = row < n ? row : row - n;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int r = col0 + j;
            if (r >= n2) break;
            double f = 0.0;
            if (row < n2) {
                const double v = sc.value(b, row, ea, r, H[j], L[j]);
                const int rr = r < n ? r : r - n;
                if (rr == cc && (r < n) != (row < n)) (r < n ? d3 : d2)[(long long)b * n + rr] = v;
                f = ax * G[(long long)rr * n + cc] * v;
                F[(long long)b * sF + (long long)r * ld + row] = f;
            }
            const unsigned m = __reduce_max_sync(0xffffffffu, cd_hi_any(f));
            if ((threadIdx.x & 31) == 0 && m) atomicMax(mx + (long long)b * mx_b + r, m);
        }
    }
};

// out_b[p = col][q = row] = alpha v + beta out, or v + omega X when X is given
struct CdEpiOut {
    static constexpr int BITS = 8;
    CdScale sc;
    double *out;
    long long ov;
    int M, N;   // |Q|, |P|
    const double *omega, *X;
    double alpha, beta;
    __device__ __forceinline__ void operator()(int b, int row, int col0, const long long (&H)[16],
                                               const long long (&L)[16]) const {
        if (row >= M) return;
        const int ea = sc.row(b, row);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int col = col0 + j;
            if (col >= N) break;
            const double v = sc.value(b, row, ea, col, H[j], L[j]);
            const long long k = (long long)col * M + row;
            double *p = out + b * ov + k;
            if (X) *p = v + omega[k] * X[b * ov + k];
            else *p = beta == 0.0 ? alpha * v : alpha * v + beta * *p;
        }
    }
};

// without exchange: G^T_b[q][r] = z_b[r] [C_Q;SC_Q][r][q], and its row maxima
__global__ void __launch_bounds__(256) cd_scale_rows_kernel(int n, int nq, const double *__restrict__ z,
                                                           const double *__restrict__ Rv, double *GT, int ld,
                                                           unsigned *mx, int mx_b) {
    const int r = blockIdx.x * 256 + threadIdx.x, q = blockIdx.y, b = blockIdx.z;
    double v = 0.0;
    if (r < 2 * n) {
        v = z[(long long)b * n + (r < n ? r : r - n)] * Rv[(long long)r * nq + q];
        GT[((long long)b * nq + q) * ld + r] = v;
    }
    const unsigned m = __reduce_max_sync(0xffffffffu, cd_hi_any(v));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(mx + (long long)b * mx_b + q, m);
}

inline long long up_to(long long x, long long m) { return (x + m - 1) / m * m; }

// the operand of nb products with `rows` rows (tile 2^rt) of K elements each
DgOperand cd_operand(bf16 *p, long long rows, long long K, int rt, long long nb) {
    return DgOperand{p, up_to(rows, 1LL << rt) * nb, up_to(K, DG_K), rt};
}

void cd_split(Ctx &c, int nb, const CdSrc &s, const DgOperand &op, const unsigned *mx, int *E) {
    const int rows_pad = (int)(op.rows_pad / nb);
    cd_split_kernel<<<dim3((unsigned)(op.Kpad / 64), rows_pad / 32, nb), 256, 0, c.stream>>>(s, rows_pad, mx, op, E);
    count_launch(c.stream, "cd_split");
    check_launch("cd_split");
}

void cd_max(Ctx &c, int nb, const CdSrc &s, int rows_pad, unsigned *mx) {
    cd_max_kernel<<<dim3(ceil_div(s.K, 64), ceil_div(s.R, 32), nb), 256, 0, c.stream>>>(s, rows_pad, mx);
    count_launch(c.stream, "cd_max");
    check_launch("cd_max");
}

template <class Epi>
void cd_gemm(Ctx &c, int family, int nb, int M, int N, int K, const DgOperand &A, bool a_shared, const DgOperand &B,
             bool b_shared, const Epi &epi) {
    const int slot = c.prof_begin(family);
    DgTiles tl{ceil_div(M, DG_M), ceil_div(N, DG_N), nb, 1, ceil_div(K, DG_K), 0, 0, 0};
    if (!a_shared) tl.a_bt = (int)(A.rows_pad / nb / DG_M);
    if (!b_shared) tl.b_bt = (int)(B.rows_pad / nb / DG_N);
    gemm_digits_tiles(c.stream, c.n_sm, tl, A, B, epi, c.d_tc_err.p);
    c.prof_end(slot, 2.0 * M * (double)N * K * nb,
               16.0 * ((double)M * K * (a_shared ? 1 : nb) + (double)N * K * (b_shared ? 1 : nb)) + 8.0 * M * (double)N * nb);
}

}  // namespace

// digits of a system's orbital blocks: [C_B;SC_B] as A and as B rows, [SC_B;C_B]^T as B rows
void Ctx::prepare_digits() {
    if (cd_ready) return;
    const int n = n_orb;
    for (int blk = 0; blk < 2; ++blk) {
        const int w = bsz(blk);
        const long long rA = up_to(2LL * n, 128), rB = up_to(2LL * n, 32), rT = up_to(w, 32);
        const long long kw = pad64(w), k2 = pad64(2LL * n);
        cd_blk[blk].reserve((size_t)DG_PLANES * (rA * kw + rB * kw + rT * k2));
        cd_eblk[blk].reserve((size_t)(rA + rB + rT));
        cd_mx.reserve((size_t)(rA + rT));
        TINCR_CUDA(cudaMemsetAsync(cd_mx.p, 0, (size_t)(rA + rT) * sizeof(unsigned), stream));
        const CdSrc st{stk(blk), 0, w, 1, 2 * n, w}, sw{swp(blk), 0, 1, w, w, 2 * n};
        cd_max(*this, 1, st, 0, cd_mx.p);
        cd_max(*this, 1, sw, 0, cd_mx.p + rA);
        cd_split(*this, 1, st, cd_stkA(blk), cd_mx.p, cd_eblk[blk].p);
        cd_split(*this, 1, st, cd_stkB(blk), cd_mx.p, cd_eblk[blk].p + rA);
        cd_split(*this, 1, sw, cd_swpT(blk), cd_mx.p + rA, cd_eblk[blk].p + rA + rB);
    }
    cd_ready = true;
}

DgOperand Ctx::cd_stkA(int blk) const { return cd_operand(cd_blk[blk].p, 2LL * n_orb, bsz(blk), 7, 1); }

DgOperand Ctx::cd_stkB(int blk) const {
    const DgOperand a = cd_stkA(blk);
    return cd_operand(a.p + DG_PLANES * a.rows_pad * a.Kpad, 2LL * n_orb, bsz(blk), 5, 1);
}

DgOperand Ctx::cd_swpT(int blk) const {
    const DgOperand b = cd_stkB(blk);
    return cd_operand(b.p + DG_PLANES * b.rows_pad * b.Kpad, bsz(blk), 2LL * n_orb, 5, 1);
}

// Bytes of workspace; half of them, what the FP64 tiles take at most (product_chunk), where the workspace has to
// grow on a device with less than four times as much free.  20 products of (H2O)128 in one chunk (1.3 GB) take
// 2.82 ms, in two 3.03.
constexpr long long CD_BUDGET = 1536LL << 20;

// Whether the digit GEMMs beat the FP64 tiles for this contraction.
bool Ctx::digits_pay(int k, int R, int S, int P, int Q, bool exch) const {
    const double n = n_orb, nr = bsz(R), ns = bsz(S), np = bsz(P), nq = bsz(Q);
    const double mac = 2.0 * n * nr * ns + 2.0 * n * np * nq + (exch ? 4.0 * n * n * (ns + nq) : 0.0);
    return contract_digits && k * mac > CD_MIN_MAC;
}

void Ctx::ao_contract_digits(int k, int R, int S, const double *V, int P, int Q, double ax, double ac, double *out,
                             double alpha, double beta, const double *Xomega) {
    tc_err_ensure();
    prepare_digits();
    const int n = n_orb, n2 = 2 * n;
    const int nr = bsz(R), ns = bsz(S), np = bsz(P), nq = bsz(Q);
    const bool exch = ax != 0.0 && lc;
    const CdSrc sR{stk(R), 0, nr, 1, n2, nr}, sS{stk(S), 0, ns, 1, n2, ns};   // [C_B;SC_B]
    const CdSrc sQ{swp(Q), 0, 1, nq, nq, n2}, sP{swp(P), 0, 1, np, np, n2};   // [SC_B;C_B]^T
    // per product: digit operands (16 bytes per padded element), FP64 results, maxima and exponents.  V, H and G
    // live one after the other and share their planes, H and G^T their FP64 results; F has its own.
    const long long rV = up_to(ns, 128), rH = up_to(n2, 32), rF = up_to(n2, 128), rG = up_to(nq, 128);
    const long long kV = pad64(nr), kH = pad64(ns), k2 = pad64(n2), ldf = up_to(n2, 4), ldh = up_to(ns, 4);
    const long long shared = std::max({rV * kV, exch ? rH * kH : 0LL, rG * k2}), el = shared + (exch ? rF * k2 : 0);
    const long long hg = std::max(n2 * ldh, nq * ldf), f64 = hg + (exch ? n2 * ldf : 0) + 3LL * n;
    const long long ints = rV + rH + rF + rG;
    const long long per = el * 16 + f64 * 8 + ints * 8;
    // chunks of equal size
    auto chunk = [&](long long budget) {
        const long long most = std::max<long long>(1, std::min<long long>(64, budget / per)), count = (k + most - 1) / most;
        return (int)((k + count - 1) / count);
    };
    int kc_max = chunk(CD_BUDGET);
    if ((size_t)(DG_PLANES * el * kc_max) > cd_pl.n || (size_t)(f64 * kc_max) > cd_f64.n) {
        size_t free_bytes = 0, total = 0;
        TINCR_CUDA(cudaMemGetInfo(&free_bytes, &total));
        if (free_bytes < 4 * (size_t)CD_BUDGET) kc_max = chunk(CD_BUDGET / 2);
    }
    cd_pl.reserve((size_t)(DG_PLANES * el * kc_max));
    cd_f64.reserve((size_t)(f64 * kc_max));
    cd_int.reserve((size_t)(2 * ints * kc_max));
    const int *eA = cd_eblk[S].p, *eB = cd_eblk[R].p + up_to(n2, 128);
    const int *eQ = cd_eblk[Q].p + up_to(n2, 128) + rH, *eP = cd_eblk[P].p + up_to(n2, 128) + rH;
    for (int c0 = 0; c0 < k; c0 += kc_max) {
        const int kc = std::min(kc_max, k - c0);
        const double *Vc = V + (long long)c0 * nr * ns;
        bf16 *pl = cd_pl.p;
        const DgOperand oV = cd_operand(pl, ns, nr, 7, kc), oG = cd_operand(pl, nq, n2, 7, kc);
        double *H = cd_f64.p, *GT = H, *d3 = H + kc * hg;
        double *d2 = d3 + (long long)kc * n, *z = d2 + (long long)kc * n, *F = z + (long long)kc * n;
        unsigned *mV = reinterpret_cast<unsigned *>(cd_int.p), *mH = mV + kc * rV, *mF = mH + kc * rH, *mG = mF + kc * rF;
        int *eV = cd_int.p + kc * ints, *eH = eV + kc * rV, *eF = eH + kc * rH, *eG = eF + kc * rF;
        TINCR_CUDA(cudaMemsetAsync(cd_int.p, 0, (size_t)(kc * ints) * sizeof(int), stream));
        // V^T: row s of product b holds V_b[r][s] over r
        const CdSrc sV{Vc, (long long)nr * ns, 1, ns, ns, nr};
        cd_max(*this, kc, sV, (int)rV, mV);
        cd_split(*this, kc, sV, oV, mV, eV);
        cd_gemm(*this, TINCR_KF_AO_TRANSFORM, kc, ns, n2, nr, oV, false, cd_stkB(R), true,
                CdEpiStore{CdScale{eV, eB, (int)rV, 0, sV, sR}, H, n2 * ldh, (int)ldh, ns, n2, mH, (int)rH});
        if (exch) {
            const DgOperand oH = cd_operand(pl, n2, ns, 5, kc), oF = cd_operand(pl + DG_PLANES * kc * shared, n2, n2, 7, kc);
            const CdSrc sH{H, n2 * ldh, ldh, 1, n2, ns}, sF{F, n2 * ldf, ldf, 1, n2, n2};
            cd_split(*this, kc, sH, oH, mH, eH);
            cd_gemm(*this, TINCR_KF_AO_EXCHANGE, kc, n2, n2, ns, cd_stkA(S), true, oH, false,
                    CdEpiF{CdScale{eA, eH, 0, (int)rH, sS, sH}, F, n2 * ldf, (int)ldf, n, d_glr_ao.p, ax, d3, d2, mF, (int)rF});
            if (ac != 0.0)
                launch_coulomb(stream, kc, n, n_atoms, d_ao_off.p, d_gamma.p, d3, d2, nullptr, F, nullptr, ac, ldf,
                               n2 * ldf, mF, (int)rF);
            cd_split(*this, kc, sF, oF, mF, eF);
            cd_gemm(*this, TINCR_KF_AO_EXCHANGE, kc, n2, nq, n2, oF, false, cd_swpT(Q), true,
                    CdEpiStore{CdScale{eF, eQ, (int)rF, 0, sF, sQ}, GT, nq * ldf, (int)ldf, n2, nq, mG, (int)rG});
        } else {
            dim3 g(ceil_div(2LL * n * 32, 256), kc);
            diag_dots_kernel<<<g, 256, 0, stream>>>(n, ns, H, ldh, n2 * ldh, stk(S), d3, d2);
            count_launch(stream, "diag_dots");
            check_launch("diag_dots");
            launch_coulomb(stream, kc, n, n_atoms, d_ao_off.p, d_gamma.p, d3, d2, z, nullptr, nullptr, ac);
            cd_scale_rows_kernel<<<dim3(ceil_div(n2, 256), nq, kc), 256, 0, stream>>>(n, nq, z, stk(Q), GT, (int)ldf, mG,
                                                                                    (int)rG);
            count_launch(stream, "cd_scale_rows");
            check_launch("cd_scale_rows");
        }
        const CdSrc sG{GT, nq * ldf, ldf, 1, nq, n2};
        cd_split(*this, kc, sG, oG, mG, eG);
        const long long o0 = (long long)c0 * np * nq;
        cd_gemm(*this, TINCR_KF_AO_TRANSFORM, kc, nq, np, n2, oG, false, cd_swpT(P), true,
                CdEpiOut{CdScale{eG, eP, (int)rG, 0, sG, sP}, out + o0, (long long)np * nq, nq, np, d_omega.p,
                         Xomega ? Xomega + o0 : nullptr, alpha, beta});
    }
    tc_err_watch();   // reported by the next sync()
}

}  // namespace tincr
