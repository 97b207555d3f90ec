// Truncated SVD on the device: svd::solver::do_svd_ptr (source/math/svd/svd.cpp:113-206) with the rank
// rule get_rank_from_truncation_error (svd.cpp:257-280) and the two-site Schmidt split
// schmidt_multisite (source/math/svd.h:189-220), for real (double) and complex (double2) matrices.
//
// Algorithm: QR-preconditioned one-sided (Hestenes) block Jacobi in FP64 (the preconditioning of Drmac & Veselic, SIAM J.
// Matrix Anal. Appl. 29 (2008) 1322-1362, without column pivoting inside the factorisations).  A is taken in its tall
// orientation (m >= n; a wide matrix as its conjugate transpose), its columns sorted by norm (few columns or too many rows
// take one factorisation or none, svd_factors):
//   A P = Q1 R1,   R1^H = Q2 R2,   Y = R2^H = U_j S V_j^H (Jacobi),   A = (Q1 U_j) S (P Q2 V_j)^H.
// The two factorisations push Y close to diagonal, so Jacobi needs 5-9 sweeps on n x n instead of 10-35 on m x n (dense
// graded spectra most: 28 -> 6 in a host model at n = 256).  Measured, graded spectrum: 512 x 512 72 -> 7.9 ms, 2048 x 2048
// 1270 -> 88 ms, complex 70 x 172 23 -> 1.4 ms, 64 x 64 3.4 -> 0.66 ms, 32 x 32 0.82 -> 0.28 ms.
//
// Jacobi: the columns of the work matrix (Y, npad columns, n padded to a multiple of 32 with zero columns) are ordered by
// norm before every sweep and grouped into blocks of 16 neighbours.  A sweep pairs every block with every other block once
// (round-robin tournament, B-1 rounds of B/2 disjoint pairs).  For one pair, a cluster of 1-4 CTAs
//   1. forms the 32 x 32 Gram matrix P^H P of the pair's 32 columns (rows streamed through shared memory,
//      DMMA products, row shares summed across the cluster),
//   2. runs one sweep of a cyclic two-sided Jacobi eigensolver on it in shared memory (16 disjoint
//      rotations per step), accumulating the unitary Q,
//   3. applies P <- P Q and V[:, pair] <- V[:, pair] Q (DMMA, row shares).
// A pair whose Gram is already diagonal to |g_ij| <= max(tol*sqrt(g_ii g_jj), floor) is skipped; the
// sweep loop stops when every pair was skipped.  The relative criterion, evaluated on freshly computed
// Gram entries, is what lets one-sided Jacobi resolve small singular values to high relative accuracy
// (Demmel & Veselic 1992), which the truncation rule at 1e-12 needs.  The absolute floor
// m eps^2 max_j ||G_j||^2 (from the previous sweep) stops the sweeps on columns that are rounding
// noise (singular values below ~eps sigma_max, which no rotation can make relatively orthogonal); an
// off-diagonal below it moves a singular value sigma by at most ~floor / sigma, the eps ||A|| level
// of LAPACK's gesdd.  Then sigma_j = ||Y_j||, U_j = Y_j / sigma_j, sorted descending.
//
// Complex rotation: for the Hermitian 2x2 block [[a, h], [conj(h), b]] with h = |h| e (|e| = 1) the
// unitary J = diag(1, conj(e)) R diag(1, e), R the real Jacobi rotation of [[a, |h|], [|h|, b]], acts as
//   col_p' = c col_p - s conj(e) col_q,   col_q' = s e col_p + c col_q
// (rows of the Gram with the conjugate coefficients); it reduces to the real rotation for e = +-1.
#include <algorithm>
#include <cmath>
#include <cooperative_groups.h>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include "matvec.cuh"
#include "runtime.cuh"
#include "svd.cuh"

namespace heff {

constexpr int JB   = 16;      // columns per block
constexpr int JP   = 2 * JB;  // columns per pair
constexpr int JTHR = 256;
constexpr int JOUTER = 60;  // outer sweeps at most

// Scalar operations of the Jacobi kernels for real and complex FP64.
template<class T>
struct JS;
template<>
struct JS<double> {
    static constexpr int ROWS = 256;            // rows of a resident tile of the pair kernel
    static constexpr int PAD = 4, PER_COPY = 2;  // leading dims == 4 (mod 16): conflict-free fragment loads; elements per 16-byte copy
    __device__ static double zero() { return 0.0; }
    __device__ static double one() { return 1.0; }
    __device__ static double fma_cj(double a, double b, double acc) { return fma(a, b, acc); }  // acc + conj(a) b
    __device__ static double fma_(double a, double b, double acc) { return fma(a, b, acc); }    // acc + a b
    __device__ static double abs2(double a) { return a * a; }
    __device__ static double absv(double a) { return fabs(a); }
    __device__ static double re(double a) { return a; }
    __device__ static double conj(double a) { return a; }
    __device__ static double mul(double a, double b) { return a * b; }
    __device__ static double axpy(double a, double x, double y) { return fma(a, x, y); }  // y + a x, a real
    __device__ static double scale(double x, double a) { return x * a; }
};
template<>
struct JS<double2> {
    static constexpr int ROWS = 128;
    static constexpr int PAD = 2, PER_COPY = 1;  // leading dims == 2 (mod 8)
    __device__ static double2 zero() { return make_double2(0.0, 0.0); }
    __device__ static double2 one() { return make_double2(1.0, 0.0); }
    __device__ static double2 fma_cj(double2 a, double2 b, double2 acc) {
        return make_double2(fma(a.x, b.x, fma(a.y, b.y, acc.x)), fma(a.x, b.y, fma(-a.y, b.x, acc.y)));
    }
    __device__ static double2 fma_(double2 a, double2 b, double2 acc) {
        return make_double2(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
    }
    __device__ static double  abs2(double2 a) { return a.x * a.x + a.y * a.y; }
    __device__ static double  absv(double2 a) {
        const double r2 = fma(a.x, a.x, a.y * a.y);
        return r2 > 1e-280 && r2 < 1e280 ? sqrt(r2) : hypot(a.x, a.y);
    }
    __device__ static double  re(double2 a) { return a.x; }
    __device__ static double2 conj(double2 a) { return make_double2(a.x, -a.y); }
    __device__ static double2 mul(double2 a, double2 b) { return cmul(a, b); }
    __device__ static double2 axpy(double a, double2 x, double2 y) { return make_double2(fma(a, x.x, y.x), fma(a, x.y, y.y)); }
    __device__ static double2 scale(double2 x, double a) { return make_double2(x.x * a, x.y * a); }
};

// Pair k of round r in the circle-method tournament over B (even) players.
__host__ __device__ inline void rr_pair(int B, int r, int k, int &p, int &q) {
    if(k == 0) {
        p = B - 1;
        q = r;
    } else {
        p = r + k < B - 1 ? r + k : r + k - (B - 1);
        q = r >= k ? r - k : r - k + (B - 1);
    }
}

__device__ inline void atomic_max_pos(double *addr, double v) {
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long *>(addr), (unsigned long long)__double_as_longlong(v));
}

// C += A B on the FP64 tensor pipe: mma.sync m16n8k4 (A fragment rows g, g+8 at column t; B at row t,
// column g; C entries (g + 8 (r >> 1), 2 t + (r & 1)), g = lane / 4, t = lane % 4).
__device__ __forceinline__ void dmma_f64(double (&c)[4], double a0, double a1, double b0) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a0), "d"(a1), "d"(b0));
}

// 2^-exponent of the larger diagonal entry: scaled by it, the squares below stay in range whatever the matrix's scale.
__device__ __forceinline__ double pair_scale(double app, double aqq) {
    const int ex = (__double2hiint(fmax(fabs(app), fabs(aqq))) >> 20) & 0x7ff;
    return __hiloint2double((2046 - min(max(ex, 1), 2045)) << 20, 0);
}
// |apq| > max(tol sqrt(app aqq), floor), all but the thresholds scaled by sc
__device__ __forceinline__ bool significant(double a, double b, double apq, double tol, double fl) {
    const double h2 = apq * apq;
    return h2 > fl * fl && h2 > tol * tol * fabs(a * b);
}
__device__ __forceinline__ bool significant(double a, double b, double2 apq, double tol, double fl) {
    const double h2 = fma(apq.x, apq.x, apq.y * apq.y);
    return h2 > fl * fl && h2 > tol * tol * fabs(a * b);
}

// Rotation that annihilates apq = |apq| e in the Hermitian 2x2 block [[app, apq], [conj(apq), aqq]]: p = 1 - cos and se = e sin
// of its angle, false when apq is not significant.  All in double precision and without a division: with x = (aqq - app) / 2,
// h = |apq| and w = sqrt(x^2 + h^2), |x| / w is the cosine of twice the angle and h / w its sine; the half-angle formulas give
// c = sqrt((1 + |x| / w) / 2) and s = h / (2 w c).  p = s^2 / (1 + c) is as right as s is, so (1 - p)^2 + s^2 = 1 holds to s^2 eps
// for tiny angles too, where 1 - c would have lost p.
template<class T>
__device__ __forceinline__ bool jacobi_rotation(double app, double aqq, T apq, double tol, double floor_abs, double &p, T &se) {
    const double sc = pair_scale(app, aqq), a = app * sc, b = aqq * sc, fl = floor_abs * sc;
    const T      z = JS<T>::scale(apq, sc);
    p  = 0.0;
    se = JS<T>::zero();
    if(!significant(a, b, z, tol, fl)) return false;
    const double x = 0.5 * (b - a), h2 = JS<T>::abs2(z);
    const double rw = rsqrt(fma(x, x, h2)), v = fma(0.5 * fabs(x), rw, 0.5), rc = rsqrt(v);  // v = c^2
    const double q = copysign(0.5 * rw * rc, x), d = fma(v, rc, 1.0);
    // 1 / (1 + c): the cubic in v with the smallest relative error on [1/2, 1] (8e-5), which does not wait for c, and two Newton steps
    double rd = fma(fma(fma(-0.094144, v, 0.323722), v, -0.49239), v, 0.762772);
    rd        = fma(rd, fma(-d, rd, 1.0), rd);
    rd        = fma(rd, fma(-d, rd, 1.0), rd);
    double       sn;
    if constexpr(std::is_same<T, double>::value) {
        se = z * q;
        sn = se;
    } else {
        se = JS<T>::scale(z, q);
        sn = h2 * rsqrt(h2) * q;
    }
    p = sn * sn * rd;
    if(p > 0.0) return true;
    se = JS<T>::zero();  // an angle below 1e-162 (or not a number): p = 0 says no rotation
    p  = 0.0;
    return false;
}
// x - (p x + c y) and x - (p x - c y): a rotation's new columns, 1 - p its cosine.  The bracket is as small as the angle, so the
// result takes one rounding of its own size (x - p x - c y from left to right takes two, complex three: orthogonality of the right
// factor 13 % worse).
__device__ __forceinline__ double  rot_sub(double x, double y, double c, double p) { return x - fma(p, x, c * y); }
__device__ __forceinline__ double  rot_add(double x, double y, double c, double p) { return x - fma(p, x, -(c * y)); }
__device__ __forceinline__ double2 rot_sub(double2 x, double2 y, double2 c, double p) {
    return make_double2(x.x - fma(p, x.x, fma(c.x, y.x, -(c.y * y.y))), x.y - fma(p, x.y, fma(c.x, y.y, c.y * y.x)));
}
__device__ __forceinline__ double2 rot_add(double2 x, double2 y, double2 c, double p) {
    return make_double2(x.x - fma(p, x.x, fma(-c.x, y.x, c.y * y.y)), x.y - fma(p, x.y, -fma(c.x, y.y, c.y * y.x)));
}

// Shared pieces of the two Jacobi kernels for P = 32 (a pair of blocks) or 64 columns on THR threads.  G and Q are P x P
// row-major with leading dim LD; a tile of rows of X or V is column-major with leading dim LDR (= rows + PAD).
template<class T, int P, int THR, int ROWS>
struct JBlock {
    using S                 = JS<T>;
    static constexpr int LD = P + S::PAD, LDR = ROWS + S::PAD, NP = P / 2, WARPS = THR / 32;
    static constexpr int TPW  = (P / 16) * (P / 8) / WARPS;  // 16 x 8 Gram tiles per warp
    static constexpr int MAT  = P * LD, TILE = P * LDR;      // elements
    static constexpr int NBLK = NP * NP / THR;               // 2 x 2 blocks per thread and step
    static_assert(TPW >= 1 && TPW * WARPS == (P / 16) * (P / 8), "Gram tiles over the warps");
    static_assert(NBLK >= 1 && THR % NP == 0, "a thread's blocks share their column pair");

    // acc += X^H X of `rows` (a multiple of 4, zero-padded) staged rows of X on the FP64 tensor pipe; complex:
    // Re = Xr^T Xr + Xi^T Xi, Im = Xr^T Xi - Xi^T Xr.  Even and odd k-steps accumulate apart: two chains of DMMAs.
    __device__ static void gram(const T *X, int rows, double (&re)[2][TPW][4], double (&im)[2][TPW][4]) {
        const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, w = threadIdx.x >> 5;
        auto      step = [&](int k4, int h) {
            const T *x = X + k4 + t;
#pragma unroll
            for(int q = 0; q < TPW; q++) {
                const int tile = w * TPW + q, mt = tile / (P / 8), nt = tile % (P / 8);
                const T   a0 = x[(mt * 16 + g) * LDR], a1 = x[(mt * 16 + g + 8) * LDR], b = x[(nt * 8 + g) * LDR];
                if constexpr(std::is_same<T, double>::value) {
                    dmma_f64(re[h][q], a0, a1, b);
                } else {
                    dmma_f64(re[h][q], a0.x, a1.x, b.x);
                    dmma_f64(im[h][q], a0.x, a1.x, b.y);
                    dmma_f64(re[h][q], a0.y, a1.y, b.y);
                    dmma_f64(im[h][q], -a0.y, -a1.y, b.x);
                }
            }
        };
        int k4 = 0;
#pragma unroll 4
        for(; k4 + 8 <= rows; k4 += 8) {
            step(k4, 0);
            step(k4 + 4, 1);
        }
        if(k4 < rows) step(k4, 0);
    }
    // element u of tile q of this thread: row, column
    __device__ static int row(int q, int u) {
        const int lane = threadIdx.x & 31, tile = (threadIdx.x >> 5) * TPW + q;
        return (tile / (P / 8)) * 16 + (lane >> 2) + 8 * (u >> 1);
    }
    __device__ static int col(int q, int u) {
        const int lane = threadIdx.x & 31, tile = (threadIdx.x >> 5) * TPW + q;
        return (tile % (P / 8)) * 8 + 2 * (lane & 3) + (u & 1);
    }
    __device__ static T make(double re, double im) {
        if constexpr(std::is_same<T, double>::value)
            return re;
        else
            return make_double2(re, im);
    }

    // Whether an off-diagonal of the Gram is significant (the same answer in every thread; a barrier), and the largest
    // diagonal entry in every thread of warp 0.
    __device__ static bool off(const T *G, int nc, double tol, double floor_abs, double &gmax) {
        bool big = false;
        for(int e = threadIdx.x; e < P * P; e += THR) {
            const int i = e / P, j = e % P;
            if(i < j && j < nc) {
                const double di = S::re(G[i * LD + i]), dj = S::re(G[j * LD + j]), sc = pair_scale(di, dj);
                big = big || significant(di * sc, dj * sc, S::scale(G[i * LD + j], sc), tol, floor_abs * sc);
            }
        }
        if(threadIdx.x < 32) {
            gmax = 0;
            for(int i = threadIdx.x; i < P; i += 32) gmax = fmax(gmax, fabs(S::re(G[i * LD + i])));
            for(int o = 16; o > 0; o >>= 1) gmax = fmax(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
        }
        return __syncthreads_or(big) != 0;
    }

    // One cyclic sweep of two-sided Jacobi on the Gram G over its first nc (even) columns, accumulating Q (set to the
    // identity here).  A step's nc / 2 disjoint rotations come from warp 0, one pair per lane, while the other warps apply
    // the previous step's rotations to Q; then every thread updates whole 2 x 2 blocks of G (rows of pair k x columns of
    // pair j, each element in exactly one block, so in place and without a barrier between the column and the row
    // rotations).  Only significant off-diagonals are rotated (half the convergence test's thresholds: the two triangles of
    // a Gram differ by rounding, and a pair that the test sees must rotate); a step without any costs one barrier.  Step s
    // pairs (nc - 1, s) and ((s + k) mod (nc - 1), (s - k) mod (nc - 1)): each thread advances its pairs by one instead of
    // evaluating the remainders.  A step takes 0.5 us (P = 32, real), most of it the chain of a rotation's operations.
    struct Pair {
        int a, b, fixed;
        __device__ Pair(int k, int nc) : a(k == 0 ? nc - 1 : k), b(k == 0 ? 0 : nc - 1 - k), fixed(k == 0) {}
        __device__ void next(int last) {  // last = nc - 2
            b = b == last ? 0 : b + 1;
            if(!fixed) a = a == last ? 0 : a + 1;
        }
    };
    __device__ static void rotate_q(T *Q, const Pair &c, T e, double p, int r0, int dr) {
        if(p == 0.0) return;
        const T ec = S::conj(e);
        for(int r = r0; r < P; r += dr) {
            T      *q = Q + r * LD;
            const T qa = q[c.a], qb = q[c.b];
            q[c.a] = rot_sub(qa, qb, ec, p);
            q[c.b] = rot_add(qb, qa, e, p);
        }
    }
    __device__ static void sweep(T *G, T *Q, T (*se_s)[NP], double (*p_s)[NP], int nc, double tol, double floor_abs) {
        const int tid = threadIdx.x, j = tid % NP, np = nc / 2;
        for(int e = tid; e < P * P; e += THR) Q[(e / P) * LD + e % P] = (e / P == e % P) ? S::one() : S::zero();
        if(tid < 2 * NP) p_s[tid / NP][tid % NP] = 0.0;  // pairs past np never rotate
        __syncthreads();
        Pair cj(j, nc), cq(j, nc), own(tid < np ? tid : 0, nc);  // block columns, Q's pair (a step behind), this lane's rotation
        int  ka[NBLK], kb[NBLK];
#pragma unroll
        for(int it = 0; it < NBLK; it++) {
            const Pair c(tid / NP + it * (THR / NP), nc);
            ka[it] = c.a, kb[it] = c.b;
        }
        bool behind = false;  // the previous step rotated: Q has not seen it
        for(int step = 0; step < nc - 1; step++) {
            const int cur = step & 1;
            bool      rot = false;
            if(tid < 32) {
                if(tid < np) {
                    double p;
                    T      se;
                    rot = jacobi_rotation<T>(S::re(G[own.a * (LD + 1)]), S::re(G[own.b * (LD + 1)]), G[own.a * LD + own.b], tol, floor_abs, p, se);
                    se_s[cur][tid] = se;
                    p_s[cur][tid]  = p;
                }
            } else if(behind) {
                rotate_q(Q, cq, se_s[cur ^ 1][j], p_s[cur ^ 1][j], (tid - 32) / NP, (THR - 32) / NP);
            }
            if(step > 0) cq.next(nc - 2);
            behind = __syncthreads_or(rot) != 0;
            if(behind) {
                const double pj = p_s[cur][j];
                const T      ej = se_s[cur][j], ejc = S::conj(ej);
#pragma unroll
                for(int it = 0; it < NBLK; it++) {
                    const int    k  = tid / NP + it * (THR / NP);
                    const double pk = p_s[cur][k];
                    if(k < np && j < np && (pk != 0.0 || pj != 0.0)) {
                        const T ek = se_s[cur][k], ekc = S::conj(ek);
                        T      *ga = G + ka[it] * LD, *gb = G + kb[it] * LD;
                        const T x00 = ga[cj.a], x01 = ga[cj.b], x10 = gb[cj.a], x11 = gb[cj.b];
                        // columns: col_a' = c col_a - s conj(e) col_b, col_b' = c col_b + s e col_a
                        const T y00 = rot_sub(x00, x01, ejc, pj), y10 = rot_sub(x10, x11, ejc, pj);
                        const T y01 = rot_add(x01, x00, ej, pj), y11 = rot_add(x11, x10, ej, pj);
                        // rows (J^H from the left): row_a' = c row_a - s e row_b, row_b' = c row_b + s conj(e) row_a
                        ga[cj.a] = rot_sub(y00, y10, ek, pk);
                        ga[cj.b] = rot_sub(y01, y11, ek, pk);
                        gb[cj.a] = rot_add(y10, y00, ekc, pk);
                        gb[cj.b] = rot_add(y11, y01, ekc, pk);
                    }
                }
                __syncthreads();
            }
            cj.next(nc - 2);
            own.next(nc - 2);
#pragma unroll
            for(int it = 0; it < NBLK; it++) {
                kb[it] = kb[it] == nc - 2 ? 0 : kb[it] + 1;
                if(tid / NP + it * (THR / NP) != 0) ka[it] = ka[it] == nc - 2 ? 0 : ka[it] + 1;
            }
        }
        if(behind) rotate_q(Q, cq, se_s[(nc - 2) & 1][j], p_s[(nc - 2) & 1][j], tid / NP, THR / NP);
        __syncthreads();
    }

    // X[row0 + r, idx[c]] = (tile Q)[r, c] for the staged rows r < rows of X (a copy of the same rows): DMMA, warp w takes
    // 16-row tiles w, w + WARPS, ..., results straight from the fragments (eight lanes on consecutive rows of a column);
    // ncols (a multiple of 32) columns.
    __device__ static void update(const T *tile, const T *Q, T *X, int64_t ldx, int64_t row0, int rows, const int *idx, int ncols) {
        const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, w = threadIdx.x >> 5;
        for(int mt = w; mt * 16 < rows; mt += WARPS) {
            const T *x = tile + mt * 16 + g;
#pragma unroll 1
            for(int nb = 0; nb < ncols / 8; nb += 4) {  // four column tiles share the row fragments
                double re[4][4], im[4][4];
#pragma unroll
                for(int q = 0; q < 4; q++)
#pragma unroll
                    for(int u = 0; u < 4; u++) re[q][u] = im[q][u] = 0.0;
#pragma unroll 4
                for(int k4 = 0; k4 < P; k4 += 4) {
                    const T a0 = x[(k4 + t) * LDR], a1 = x[(k4 + t) * LDR + 8];
#pragma unroll
                    for(int q = 0; q < 4; q++) {
                        const T b = Q[(k4 + t) * LD + (nb + q) * 8 + g];
                        if constexpr(std::is_same<T, double>::value) {
                            dmma_f64(re[q], a0, a1, b);
                        } else {
                            dmma_f64(re[q], a0.x, a1.x, b.x);
                            dmma_f64(im[q], a0.x, a1.x, b.y);
                            dmma_f64(re[q], -a0.y, -a1.y, b.y);
                            dmma_f64(im[q], a0.y, a1.y, b.x);
                        }
                    }
                }
#pragma unroll
                for(int q = 0; q < 4; q++)
#pragma unroll
                    for(int u = 0; u < 4; u++) {
                        const int r = mt * 16 + g + 8 * (u >> 1), c = (nb + q) * 8 + 2 * t + (u & 1);
                        if(r < rows) X[row0 + r + ldx * (int64_t)idx[c]] = make(re[q][u], im[q][u]);
                    }
            }
        }
    }
    // Rows [row0, row0 + rows) of the columns idx of X into tile (columns past ncols and rows up to the next multiple of 16
    // as zeros), a column per warp in 16-byte copies (row0, ldx and X's address are even multiples of an element; a copy's
    // second row may be the zero row that pads an odd number of rows); complete after stage_wait and a barrier.
    __device__ static void stage(T *tile, const T *X, int64_t ldx, int64_t row0, int rows, const int *idx, int ncols) {
        const int rp = (rows + 15) / 16 * 16, lane = threadIdx.x & 31;
        for(int c = threadIdx.x >> 5; c < P; c += WARPS) {
            const T *src = X + row0 + ldx * (int64_t)idx[c];
            for(int r = lane * S::PER_COPY; r < rp; r += 32 * S::PER_COPY) {
                const bool v = r < rows && c < ncols;
                cp_async<16>(smem_u32(tile + r + c * LDR), v ? src + r : X, v);
            }
        }
        cp_async_commit();
    }
    __device__ static void stage_wait() { cp_async_wait<0>(); }
};

// One round of the block Jacobi sweep.  A pair is handled by a cluster of CL CTAs (blockIdx.x = pair * CL + rank):
// each forms the Gram of its share of the rows and sends it to every CTA of the cluster through distributed shared memory;
// every CTA sums the partials in rank order (the same full Gram everywhere), runs the small Jacobi on it (the same Q
// everywhere, no broadcast) and updates its share of the rows of G and V.  CL = 1: a plain launch, one CTA per pair.  The
// cluster barrier is reached by every CTA; the early exit comes after it.  A share of at most JS::ROWS rows of G stays in
// shared memory from the Gram to the update; the share of V loads during the small Jacobi.
// Bound by the latency of the small Jacobi's 31 dependent steps: at 512 x 512 (CL = 4) 35 of 53 thousand clocks, the Gram 5,
// its sum over the cluster 3.5, the updates 7.6 (27 us a round; 75 us before: 47 thousand for steps of three barriers and a
// chain of divisions and square roots, bank conflicts in every fragment load, the Gram read back element by element).
template<class T>
using JPairBlock = JBlock<T, JP, JTHR, JS<T>::ROWS>;
constexpr int JCL = 4;  // CTAs per pair at most
template<class T>
constexpr size_t jacobi_round_bytes() {
    using JK = JPairBlock<T>;
    static_assert(JK::MAT + JK::TILE >= JCL * JK::MAT, "the partial Grams fit Q and the tile of V");
    return sizeof(T) * (size_t)(2 * JK::MAT + 2 * JK::TILE);
}
template<class T>
__global__ void __launch_bounds__(JTHR) jacobi_round_kernel(T *__restrict__ G, int64_t ldg, int m, T *__restrict__ V, int64_t ldv, int nv, int B,
                                                           int round, double tol, double floor_abs, const int *__restrict__ colmap,
                                                           double *__restrict__ gmax_out, int *__restrict__ rotated, int CL) {
    grid_wait();
    if(CL > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");  // met before the first remote store
    using S  = JS<T>;
    using JK = JPairBlock<T>;
    constexpr int RC = S::ROWS;
    extern __shared__ __align__(16) unsigned char jr_smem[];
    T                *sG = reinterpret_cast<T *>(jr_smem), *sT = sG + JK::MAT, *sQ = sT + JK::TILE, *sV = sQ + JK::MAT;
    T                *sPart = sQ;  // CL partial Grams, before Q and the tile of V are used
    __shared__ T      s_se[2][JP / 2];
    __shared__ double s_p[2][JP / 2];
    __shared__ int    s_idx[JP];

    int       p, q;
    const int rank = (int)(blockIdx.x % CL);
    rr_pair(B, round, (int)(blockIdx.x / CL), p, q);
    const int tid = threadIdx.x;
    if(tid < JP) s_idx[tid] = colmap[(tid < JB) ? p * JB + tid : q * JB + (tid - JB)];
    __syncthreads();

    // ---- 1. Gram matrix of the 32 columns over this CTA's rows [ga, gb) (shares of whole 16-row tiles)
    auto share = [&](int rows, int r) { return min(rows, (rows + 16 * CL - 1) / (16 * CL) * 16 * r); };
    const int ga = share(m, rank), gb = share(m, rank + 1);
    double    re[2][JK::TPW][4] = {}, im[2][JK::TPW][4] = {};
    for(int r0 = ga; r0 < gb; r0 += RC) {
        const int rows = min(RC, gb - r0);
        if(r0 > ga) __syncthreads();  // the previous tile has been read
        JK::stage(sT, G, ldg, r0, rows, s_idx, JP);
        JK::stage_wait();
        __syncthreads();
        JK::gram(sT, (rows + 3) / 4 * 4, re, im);
    }
    if(CL == 1) {
#pragma unroll
        for(int k = 0; k < JK::TPW; k++)
#pragma unroll
            for(int u = 0; u < 4; u++) sG[JK::row(k, u) * JK::LD + JK::col(k, u)] = JK::make(re[0][k][u] + re[1][k][u], im[0][k][u] + im[1][k][u]);
    } else {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        T *mine = sPart + rank * JK::MAT;
#pragma unroll
        for(int k = 0; k < JK::TPW; k++)
#pragma unroll
            for(int u = 0; u < 4; u++) mine[JK::row(k, u) * JK::LD + JK::col(k, u)] = JK::make(re[0][k][u] + re[1][k][u], im[0][k][u] + im[1][k][u]);
        __syncthreads();
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");  // every CTA has started: its shared memory may be written
        constexpr int PC = S::PER_COPY;  // 16 bytes a store, whole rows in order
        for(int r = 1; r < CL; r++) {
            const int to  = (rank + r) % CL;
            T        *dst = cluster.map_shared_rank(sPart, to) + rank * JK::MAT;
            for(int e = tid; e < JP * JP / PC; e += JTHR) {
                const int at = (e / (JP / PC)) * JK::LD + e % (JP / PC) * PC;
                *reinterpret_cast<double2 *>(dst + at) = *reinterpret_cast<const double2 *>(mine + at);
            }
        }
        cluster.sync();
        for(int e = tid; e < JP * JP; e += JTHR) {
            const int at = (e / JP) * JK::LD + e % JP;
            T         v  = sPart[at];
            for(int r = 1; r < CL; r++) v = S::axpy(1.0, sPart[r * JK::MAT + at], v);
            sG[at] = v;
        }
    }
    __syncthreads();

    // ---- off-diagonal test of the fresh Gram, and the largest squared column norm (the next sweep's floor)
    double     gm  = 0;
    const bool big = JK::off(sG, JP, tol, floor_abs, gm);
    if(tid == 0 && rank == 0) atomic_max_pos(gmax_out, gm);
    if(!big) return;  // uniform across the CTA and the cluster (the same Gram everywhere)
    if(tid == 0 && rank == 0) atomicAdd(rotated, 1);

    // ---- 2. one sweep of two-sided Jacobi (the outer sweep re-checks every pair on a freshly computed Gram matrix;
    //      measured on 1024^2 and 2048^2: one inner sweep costs at most a few more outer sweeps and halves the time
    //      against eight)
    const int va = share(nv, rank), vb = share(nv, rank + 1);
    if(vb - va <= RC) JK::stage(sV, V, ldv, va, vb - va, s_idx, JP);
    JK::sweep(sG, sQ, s_se, s_p, JP, 0.5 * tol, 0.5 * floor_abs);

    // ---- 3. apply Q to this CTA's share of the pair's columns of G (m rows) and V (nv rows)
    for(int pass = 0; pass < 2; pass++) {
        T            *X    = pass == 0 ? G : V, *tile = pass == 0 ? sT : sV;
        const int64_t ldx  = pass == 0 ? ldg : ldv;
        const int     ra = pass == 0 ? ga : va, rb = pass == 0 ? gb : vb;
        for(int r0 = ra; r0 < rb; r0 += RC) {
            const int rows = min(RC, rb - r0);
            if(rb - ra > RC) {
                __syncthreads();  // the previous tile has been read
                JK::stage(tile, X, ldx, r0, rows, s_idx, JP);
            }
            JK::stage_wait();
            __syncthreads();
            JK::update(tile, sQ, X, ldx, r0, rows, s_idx, JP);
        }
    }
}

// Small matrices (at most P = 32 or 64 columns): one CTA runs every sweep on all columns as one block -- Gram, one cyclic
// Jacobi sweep over the round-robin tournament of the first nc (even) columns, update -- with no host round trip between
// sweeps, and the copies before and the norms after as well: at these sizes every further launch or synchronisation costs
// as much as a sweep.  Up to JW_ROWS rows, X and V stay in shared memory (three tiles: a product goes to the free one);
// longer X, and complex X of 64 columns, pass through one tile per JW_ROWS rows of global memory.
// A (m x n; adjoint: n x m, read as its conjugate transpose) may be X itself; X (m x P) and V (P x P) receive the rotated
// columns and the rotations, sig the column norms, *sweeps_out the number of sweeps run (max_sweeps when the last one
// still rotated).
constexpr int JW_P = 64, JW_ROWS = 64;
constexpr int jw_thr(int P) { return P == 32 ? 256 : 512; }
template<class T, int P>
using JWholeBlock = JBlock<T, P, jw_thr(P), JW_ROWS>;
template<class T, int P>
constexpr bool jw_resident() {
    return sizeof(T) == 8 || P == 32;
}
template<class T, int P>
constexpr size_t jacobi_whole_bytes() {
    return sizeof(T) * (size_t)(2 * JWholeBlock<T, P>::MAT + (jw_resident<T, P>() ? 3 : 1) * JWholeBlock<T, P>::TILE);
}
template<class T, int P>
__global__ void __launch_bounds__(jw_thr(P), 1) jacobi_whole_kernel(const T *A, int64_t lda, int adjoint, T *X, int64_t ldx, int m, int n, T *V, double tol,
                                                                   int max_sweeps, double *__restrict__ sig, int *__restrict__ sweeps_out) {
    grid_wait();
    using S  = JS<T>;
    using JK = JWholeBlock<T, P>;
    constexpr int THR = jw_thr(P);
    extern __shared__ __align__(16) unsigned char jw_smem[];
    T                *sG = reinterpret_cast<T *>(jw_smem), *sQ = sG + JK::MAT, *sT = sQ + JK::MAT;
    __shared__ T      s_se[2][P / 2];
    __shared__ double s_p[2][P / 2], s_gmax;
    __shared__ int    s_idx[P];
    const int         tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double      eps = 2.220446049250313e-16;
    const bool        res = jw_resident<T, P>() && m <= JW_ROWS;
    const int         nc  = (n + 1) / 2 * 2;  // padded columns are zero and never rotate
    T                *bx = sT, *bv = sT + JK::TILE, *bf = sT + 2 * JK::TILE;  // resident: X, V and the free tile
    if(tid < P) s_idx[tid] = tid;
    auto src = [&](int r, int c) { return (r < m && c < n) ? (adjoint ? S::conj(A[c + lda * (int64_t)r]) : A[r + lda * (int64_t)c]) : S::zero(); };
    if(res) {
        for(int e = tid; e < JK::TILE; e += THR) {
            const int c = e / JK::LDR, r = e % JK::LDR;
            bx[e] = src(r, c);
            bv[e] = r == c ? S::one() : S::zero();
            bf[e] = S::zero();
        }
    } else {
        for(int c = warp; c < P; c += THR / 32) {
            if(A != X)
                for(int64_t r = lane; r < ldx; r += 32) X[r + ldx * c] = src((int)r, c);
            for(int r = lane; r < P; r += 32) V[r + P * c] = r == c ? S::one() : S::zero();
        }
    }
    double floor_abs = 0.0;  // first sweep: relative criterion only
    int    done      = max_sweeps;
    for(int sweep = 0; sweep < max_sweeps; sweep++) {
        double re[2][JK::TPW][4] = {}, im[2][JK::TPW][4] = {};
        __syncthreads();
        if(res) {
            JK::gram(bx, (m + 3) / 4 * 4, re, im);
        } else {
            for(int r0 = 0; r0 < m; r0 += JW_ROWS) {
                const int rows = min(JW_ROWS, m - r0);
                if(r0 > 0) __syncthreads();
                JK::stage(sT, X, ldx, r0, rows, s_idx, P);
                JK::stage_wait();
                __syncthreads();
                JK::gram(sT, (rows + 3) / 4 * 4, re, im);
            }
        }
#pragma unroll
        for(int k = 0; k < JK::TPW; k++)
#pragma unroll
            for(int u = 0; u < 4; u++) sG[JK::row(k, u) * JK::LD + JK::col(k, u)] = JK::make(re[0][k][u] + re[1][k][u], im[0][k][u] + im[1][k][u]);
        __syncthreads();
        double     gm  = 0;
        const bool big = JK::off(sG, nc, tol, floor_abs, gm);
        if(!big) {
            done = sweep + 1;
            break;
        }
        if(tid == 0) s_gmax = gm;
        JK::sweep(sG, sQ, s_se, s_p, nc, 0.5 * tol, 0.5 * floor_abs);
        if(res) {
            JK::update(bx, sQ, bf, JK::LDR, 0, m, s_idx, P);
            __syncthreads();
            JK::update(bv, sQ, bx, JK::LDR, 0, P, s_idx, P);
            T *t = bx;
            bx = bf, bf = bv, bv = t;  // the free tile holds V's old rows: its rows past m are zeroed before it takes X
            __syncthreads();
            for(int e = tid; e < JK::TILE; e += THR)
                if(e % JK::LDR >= m) bf[e] = S::zero();
        } else {
            for(int pass = 0; pass < 2; pass++) {
                T            *B   = pass == 0 ? X : V;
                const int64_t ldb = pass == 0 ? ldx : P;
                const int     all = pass == 0 ? m : P;
                for(int r0 = 0; r0 < all; r0 += JW_ROWS) {
                    const int rows = min(JW_ROWS, all - r0);
                    __syncthreads();
                    JK::stage(sT, B, ldb, r0, rows, s_idx, P);
                    JK::stage_wait();
                    __syncthreads();
                    JK::update(sT, sQ, B, ldb, r0, rows, s_idx, P);
                }
            }
        }
        __syncthreads();
        floor_abs = (double)m * eps * eps * s_gmax;
    }
    __syncthreads();
    for(int c = warp; c < P; c += THR / 32) {
        double acc = 0.0;
        for(int r = lane; r < m; r += 32) {
            const T v = res ? bx[r + c * JK::LDR] : X[r + ldx * (int64_t)c];
            if(res) X[r + ldx * (int64_t)c] = v;
            acc += S::abs2(v);
        }
        for(int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if(lane == 0) sig[c] = sqrt(acc);
        if(res)
            for(int r = lane; r < P; r += 32) V[r + P * c] = bv[r + c * JK::LDR];
    }
    if(tid == 0) *sweeps_out = done;
}

// sigma_j = ||G_j||_2 (column norms), one warp per column.
template<class T>
__global__ void col_norms_kernel(const T *__restrict__ G, int64_t ldg, int m, int n, double *__restrict__ sig) {
    grid_wait();
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
    if(w >= n) return;
    double acc = 0;
    for(int i = lane; i < m; i += 32) acc += JS<T>::abs2(G[i + ldg * (int64_t)w]);
    for(int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if(lane == 0) sig[w] = sqrt(acc);
}

// Stable descending order of the column norms: ord[rank of column i] = i (a NaN sorts last).
__global__ void col_order_kernel(const double *__restrict__ sig, int n, int *__restrict__ ord) {
    grid_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const double a = sig[i] >= 0 ? sig[i] : -1.0;
    int          r = 0;
    for(int j = 0; j < n; j++) {
        const double b = sig[j] >= 0 ? sig[j] : -1.0;
        r += (b > a || (b == a && j < i)) ? 1 : 0;
    }
    ord[r] = i;
}

// G (rows x npad, leading dim ldg, zero-padded) = A (m x n, leading dim lda) with its columns in the order ord, or A^H
// (n x m) without a reordering.  ord may be nullptr (identity).
template<class T>
__global__ void copy_pad_kernel(const T *__restrict__ A, int64_t lda, int rows, int cols, T *__restrict__ G, int64_t ldg, int npad,
                                const int *__restrict__ ord) {
    grid_wait();
    const int64_t tot = (int64_t)ldg * npad;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e % ldg, c = e / ldg;
        G[e]            = (r < rows && c < cols) ? A[r + lda * (ord ? ord[c] : c)] : JS<T>::zero();
    }
}
// Y (ldy x ncol, zero where r >= rows or c >= cols) = X^H (or its upper triangle's, UPPER), 32 x 32 tiles through shared
// memory, X read and Y written along columns.
template<class T, bool UPPER>
__global__ void __launch_bounds__(256) adjoint_kernel(const T *__restrict__ X, int64_t ldx, int xrows, int xcols, T *__restrict__ Y, int64_t ldy, int yrows,
                                                     int ycols) {
    grid_wait();
    __shared__ T tile[32][33];
    const int    x0 = blockIdx.x * 32, y0 = blockIdx.y * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5;  // Y rows from y0, columns from x0
    for(int c = w; c < 32; c += 8) {
        const int r = x0 + lane, k = y0 + c;  // X[r, k]
        tile[c][lane] = (r < xrows && k < xcols && (!UPPER || r <= k)) ? X[r + ldx * (int64_t)k] : JS<T>::zero();
    }
    __syncthreads();
    for(int c = w; c < 32; c += 8)
        if(y0 + lane < yrows && x0 + c < ycols) Y[(y0 + lane) + ldy * (int64_t)(x0 + c)] = JS<T>::conj(tile[lane][c]);
}

template<class T>
__global__ void eye_kernel(T *__restrict__ V, int64_t ldv, int npad) {
    grid_wait();
    const int64_t tot = (int64_t)ldv * npad;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x)
        V[e] = (e % ldv == e / ldv) ? JS<T>::one() : JS<T>::zero();
}

// S[i] = sig[perm[i]]; left[r, i] = W[r, perm[i]] / S[i] (0 for S[i] = 0), r < rows, and 0 up to lrows; right[r, i] =
// V[r, perm[i]], r < n.  LADJ / RADJ: the conjugate transpose of left / right instead (k x lrows, k x n, leading dim k).
template<class T, bool LADJ, bool RADJ>
__global__ void take_columns_kernel(const T *__restrict__ W, int64_t ldw, int rows, const T *__restrict__ V, int64_t ldv, int n, const int *__restrict__ perm,
                                    const double *__restrict__ sig, int k, double *__restrict__ Sout, T *__restrict__ left, int64_t ldl, int lrows,
                                    T *__restrict__ right, int64_t ldr) {
    grid_wait();
    const int64_t tl = (int64_t)lrows * k, tot = tl + (int64_t)n * k;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const bool    lt = e < tl;
        const int64_t f  = lt ? e : e - tl;
        const bool    adj = lt ? LADJ : RADJ;
        const int64_t len = lt ? lrows : n, i = adj ? f % k : f / len, r = adj ? f / k : f % len;
        const int     j = perm[i];
        T             v;
        if(lt) {
            const double sj = sig[j];
            v = r < rows && sj > 0 ? JS<T>::scale(W[r + ldw * (int64_t)j], 1.0 / sj) : JS<T>::zero();
            if(r == 0) Sout[i] = sj;
        } else {
            v = V[r + ldv * (int64_t)j];
        }
        if(adj)
            (lt ? left : right)[i + (int64_t)k * r] = JS<T>::conj(v);
        else if(lt)
            left[r + ldl * i] = v;
        else
            right[r + ldr * i] = v;
    }
}
// B (k x n, leading dim k)[i, ord[c]] = conj(X[c, i]);  ord may be nullptr (identity)
template<class T>
__global__ void adjoint_rows_kernel(const T *__restrict__ X, int64_t ldx, int n, int k, const int *__restrict__ ord, T *__restrict__ B) {
    grid_wait();
    const int64_t tot = (int64_t)n * k;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e / k, i = e % k;
        B[i + (int64_t)k * (ord ? ord[c] : c)] = JS<T>::conj(X[c + ldx * i]);
    }
}
// out[ord[c], i] = X[c, i]
template<class T>
__global__ void scatter_rows_kernel(const T *__restrict__ X, int64_t ldx, int n, int k, const int *__restrict__ ord, T *__restrict__ out, int64_t ldo) {
    grid_wait();
    const int64_t tot = (int64_t)n * k;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / n, c = e % n;
        out[ord[c] + ldo * i] = X[c + ldx * i];
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Householder QR in panels of 16 columns (LAPACK's ?geqr2 / ?larft conventions: H_j = I - tau_j v_j v_j^H, Q = H_0 H_1 ... =
// I - V T V^H, beta real).  The factors stay in place: R on and above the diagonal, V below it.
constexpr int QW = 16;

// Sum of d[0..15] over the warp by exchanging halves: 16 (real) or 32 (complex) shuffle pairs instead of 80 or 160; the
// lanes 2 i and 2 i + 1 end with the sum of d[i].
template<class T>
__device__ __forceinline__ T qr_shfl(T v, int o);
template<>
__device__ __forceinline__ double qr_shfl(double v, int o) {
    return __shfl_xor_sync(0xffffffffu, v, o);
}
template<>
__device__ __forceinline__ double2 qr_shfl(double2 v, int o) {
    return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ double  qr_add(double a, double b) { return a + b; }
__device__ __forceinline__ double2 qr_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
template<class T>
__device__ __forceinline__ T qr_warp_sum16(T (&d)[QW]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for(int o = 16, h = 8; o > 1; o >>= 1, h >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for(int i = 0; i < 8; i++)
            if(i < h) {
                const T snd = up ? d[i] : d[i + h], own = up ? d[i + h] : d[i];
                d[i]        = qr_add(own, qr_shfl(snd, o));
            }
    }
    return qr_add(d[0], qr_shfl(d[0], 1));
}

// Factors the panel of columns [j0, j0 + w), rows [j0, M), of G, and forms its T (QW x QW, column-major).  Each thread keeps
// RPT rows of the panel in registers.  A step needs one reduction: the products x^H a_c of the pivot column with every
// column of the panel give its norm, the coefficients of the update of the later columns and (c < j, where a_c holds v_c)
// the column of V^H V that T's recurrence takes.  The last warp of the CTA holds no rows: it turns the sums into
// coefficients and carries T along while the others update.  CL CTAs of a cluster share a long panel's rows (their sums
// are exchanged through distributed shared memory and added in rank order by every CTA).  The step loop is not unrolled:
// the pivot column is always register column 0 and the columns rotate by one after each step (unrolled, every instruction
// of the kernel ran once and the fetches bound it: 70 us a panel of 512 rows, now 23).
template<class T>
struct QrPanel {
    static constexpr int RPT      = sizeof(T) == 16 ? 2 : 3;
    static constexpr int THR_MAX  = 224;                // threads with rows (with the coefficient warp 256: 255 registers each)
    static constexpr int THR_MIN  = 96;
    static constexpr int ROWS_MAX = 8 * RPT * THR_MAX;  // rows of a panel over a cluster of 8
};
template<class T>
__global__ void __launch_bounds__(QrPanel<T>::THR_MAX + 32, 1) qr_panel_kernel(T *__restrict__ G, int64_t ldg, int M, int j0, int w, T *__restrict__ Tout, int CL) {
    grid_wait();
    if(CL > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");  // met before the first remote store
    using S           = JS<T>;
    constexpr int RPT = QrPanel<T>::RPT;
    __shared__ T      s_red[QrPanel<T>::THR_MAX / 32][QW];
    __shared__ T      s_row[QW];           // row j of the panel before step j (rank 0's)
    __shared__ T      s_cl[2][8][QW + QW]; // per rank: its sums, and (rank 0) row j
    __shared__ T      s_f[QW], s_g[QW], s_inv;
    __shared__ double s_beta;
    const int         thr = (int)blockDim.x - 32, nw = thr / 32, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int         rank = (int)blockIdx.x, rows = M - j0;
    const bool        ctl = tid >= thr;  // the coefficient warp: lane l stands for column l
    const int         lr0 = rank * RPT * thr + tid;  // local row of slot i: lr0 + i * thr
    // register column c is panel column (j + c) % QW before step j (coefficient warp: a[0] is row `lane` of T, unrotated)
    T a[RPT][QW];
#pragma unroll
    for(int i = 0; i < RPT; i++)
#pragma unroll
        for(int c = 0; c < QW; c++) a[i][c] = (!ctl && lr0 + i * thr < rows && c < w) ? G[(j0 + lr0 + i * thr) + ldg * (int64_t)(j0 + c)] : S::zero();

#pragma unroll 1
    for(int j = 0; j < w; j++) {  // registers of columns past w hold zeros and change nothing
        if(!ctl) {
            T d[QW];
#pragma unroll
            for(int c = 0; c < QW; c++) d[c] = S::zero();
#pragma unroll
            for(int i = 0; i < RPT; i++) {
                const T x = (lr0 + i * thr >= j) ? a[i][0] : S::zero();
#pragma unroll
                for(int c = 0; c < QW; c++) d[c] = S::fma_cj(x, a[i][c], d[c]);
            }
            const T sum = qr_warp_sum16(d);
            if((lane & 1) == 0) s_red[warp][lane >> 1] = sum;
            if(lr0 == j) {
#pragma unroll
                for(int c = 0; c < QW; c++) s_row[c] = a[0][c];
            }
        }
        __syncthreads();
        const int slot = (lane - j) & (QW - 1);  // register column of panel column `lane`
        T         tot = S::zero(), ajc = S::zero(), piv = S::zero(), alpha = S::zero();  // this column's and the pivot's sums, row j
        if(ctl) {
            T u[QrPanel<T>::THR_MAX / 32], v[QrPanel<T>::THR_MAX / 32];
#pragma unroll
            for(int q = 0; q < QrPanel<T>::THR_MAX / 32; q++) {
                u[q] = q < nw ? s_red[q][slot] : S::zero();
                v[q] = q < nw ? s_red[q][0] : S::zero();
            }
#pragma unroll
            for(int q = 0; q < QrPanel<T>::THR_MAX / 32; q++) tot = qr_add(tot, u[q]), piv = qr_add(piv, v[q]);
            ajc   = s_row[slot];
            alpha = s_row[0];
        }
        if(CL > 1) {
            namespace cg = cooperative_groups;
            cg::cluster_group cluster = cg::this_cluster();
            if(j == 0) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");  // every CTA has started
            if(ctl && lane < QW)
                for(int q = 0; q < CL; q++) {
                    T *dst    = cluster.map_shared_rank(&s_cl[j & 1][rank][0], q);
                    dst[lane] = tot;
                    if(rank == 0) dst[QW + lane] = ajc;
                }
            cluster.sync();
            if(ctl) {
                tot = piv = S::zero();
                for(int q = 0; q < CL; q++) tot = qr_add(tot, s_cl[j & 1][q][lane & (QW - 1)]), piv = qr_add(piv, s_cl[j & 1][q][j]);
                ajc   = s_cl[j & 1][0][QW + (lane & (QW - 1))];
                alpha = s_cl[j & 1][0][QW + j];
            }
        }
        T tau = S::zero(), z = S::zero();
        if(ctl) {
            // v = (x - beta e_j) inv, v_j = 1; w_c = v^H a_c = conj(inv) (x^H a_c - beta a_jc); a_c -= conj(tau) w_c v
            const double sig2 = S::re(piv);
            double beta = sig2;  // zero column: 0; a NaN stays one
            T      inv = S::zero(), g = S::zero(), f = S::zero();
            if(sig2 > 0) {
                const double rs = rsqrt(sig2), nrm = sig2 * rs, ar = S::re(alpha);
                beta            = ar >= 0 ? -nrm : nrm;
                const double ib = ar >= 0 ? -rs : rs;
                T            wc;
                if constexpr(std::is_same<T, double>::value) {
                    inv = 1.0 / (alpha - beta);
                    tau = (beta - alpha) * ib;
                    wc  = (tot - beta * ajc) * inv;
                    g   = tau * wc;
                    f   = g * inv;
                } else {  // |Im alpha| <= |alpha - beta|: the quotient keeps the square in range
                    const double dr = ar - beta, q = alpha.y / dr, den = 1.0 / (dr * fma(q, q, 1.0));
                    inv = make_double2(den, -q * den);
                    tau = make_double2((beta - ar) * ib, -alpha.y * ib);
                    wc  = cmul(S::conj(inv), make_double2(fma(-beta, ajc.x, tot.x), fma(-beta, ajc.y, tot.y)));
                    g   = cmul(S::conj(tau), wc);
                    f   = cmul(g, inv);
                }
                if(lane < j) {
                    z = S::conj(wc);  // v_lane^H v_j; finished columns are not updated
                    f = g = S::zero();
                }
            }
            if(lane < QW) s_f[slot] = f, s_g[slot] = g;
            if(lane == 0) s_inv = inv, s_beta = beta;
        }
        __syncthreads();
        if(ctl) {
            // T[c, j] = -tau_j sum_{c <= k < j} T[c, k] z_k, T[j, j] = tau_j (z_k = 0 for k >= j)
            T acc[2] = {S::zero(), S::zero()};
#pragma unroll
            for(int k = 0; k < QW; k++) {
                T zk;
                if constexpr(std::is_same<T, double>::value)
                    zk = __shfl_sync(0xffffffffu, z, k);
                else
                    zk = make_double2(__shfl_sync(0xffffffffu, z.x, k), __shfl_sync(0xffffffffu, z.y, k));
                acc[k & 1] = S::fma_(a[0][k], zk, acc[k & 1]);
            }
            const T tj = lane < j ? S::scale(S::mul(tau, qr_add(acc[0], acc[1])), -1.0) : (lane == j ? tau : S::zero());
#pragma unroll
            for(int k = 0; k < QW; k++)
                if(k == j) a[0][k] = tj;
        } else {
            const T inv = s_inv;
            T       f[QW];
#pragma unroll
            for(int c = 1; c < QW; c++) f[c] = s_f[c];
#pragma unroll
            for(int i = 0; i < RPT; i++) {
                const int lr = lr0 + i * thr;
                T         v  = a[i][0];
                if(lr > j) {
                    const T x = S::scale(v, -1.0);
#pragma unroll
                    for(int c = 1; c < QW; c++) a[i][c] = S::fma_(x, f[c], a[i][c]);
                    v = S::mul(v, inv);
                } else if(lr == j) {
#pragma unroll
                    for(int c = 1; c < QW; c++) a[i][c] = S::axpy(-1.0, s_g[c], a[i][c]);
                    if constexpr(std::is_same<T, double>::value)
                        v = s_beta;
                    else
                        v = make_double2(s_beta, 0.0);
                }
#pragma unroll
                for(int c = 1; c < QW; c++) a[i][c - 1] = a[i][c];
                a[i][QW - 1] = v;
            }
        }
    }
    if(!ctl) {
#pragma unroll
        for(int i = 0; i < RPT; i++)
#pragma unroll
            for(int c = 0; c < QW; c++) {
                const int pc = (c + w) & (QW - 1);  // the columns have been rotated w times
                if(lr0 + i * thr < rows && pc < w) G[(j0 + lr0 + i * thr) + ldg * (int64_t)(j0 + pc)] = a[i][c];
            }
    } else if(rank == 0 && lane < QW) {
#pragma unroll
        for(int c = 0; c < QW; c++) Tout[lane + QW * c] = a[0][c];
    }
    if(CL > 1) cooperative_groups::this_cluster().sync();  // no CTA leaves while its sums may be written
}

// A[r0 .. M, c0 .. c0 + nc) <- (I - V T V^H) A, or with T^H (ADJ), for the panel at column j0 of G (V unit lower trapezoidal
// below the diagonal, r0 = j0).  One CTA per 16 columns of A: W = V^H A over the rows (DMMA, warps share the rows), T W in
// shared memory, A -= V (T W).  The fragments come straight from L2.
template<class T, bool ADJ>
__global__ void __launch_bounds__(256) qr_apply_kernel(const T *__restrict__ G, int64_t ldg, int M, int j0, const T *__restrict__ Tm, T *__restrict__ A,
                                                      int64_t lda, int nc) {
    grid_wait();
    using S = JS<T>;
    constexpr bool C = !std::is_same<T, double>::value;
    __shared__ T     sW[8][QW][QW + 1], sX[QW][QW + 1], sT[QW][QW + 1];
    const int        tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const int        c0 = blockIdx.x * QW, rows = M - j0;
    const T         *Vp = G + j0 + ldg * (int64_t)j0;
    T               *Ap = A + j0 + lda * (int64_t)c0;
    const int        cw = min(QW, nc - c0);
    // V[r, c] of the panel: unit diagonal, zero above
    auto v = [&](int r, int c) -> T {
        if(r >= rows || r < c) return S::zero();
        return r == c ? S::one() : Vp[r + ldg * (int64_t)c];
    };
    sT[tid / QW][tid % QW] = Tm[tid / QW + QW * (tid % QW)];
    double wr[2][4] = {}, wi[2][4] = {};
#pragma unroll 4
    for(int r0 = 4 * w; r0 < rows; r0 += 32) {
        const int r  = r0 + t;
        const T   a0 = v(r, g), a1 = v(r, g + 8);
#pragma unroll
        for(int q = 0; q < 2; q++) {
            const int c = q * 8 + g;
            const T   b = (r < rows && c < cw) ? Ap[r + lda * (int64_t)c] : S::zero();
            if constexpr(!C) {
                dmma_f64(wr[q], a0, a1, b);
            } else {  // conj(V) A
                dmma_f64(wr[q], a0.x, a1.x, b.x);
                dmma_f64(wi[q], a0.x, a1.x, b.y);
                dmma_f64(wr[q], a0.y, a1.y, b.y);
                dmma_f64(wi[q], -a0.y, -a1.y, b.x);
            }
        }
    }
#pragma unroll
    for(int q = 0; q < 2; q++)
#pragma unroll
        for(int u = 0; u < 4; u++) {
            T &o = sW[w][g + 8 * (u >> 1)][q * 8 + 2 * t + (u & 1)];
            if constexpr(!C)
                o = wr[q][u];
            else
                o = make_double2(wr[q][u], wi[q][u]);
        }
    __syncthreads();
    const int wi0 = tid / QW, wj = tid % QW;
    T         sum = sW[0][wi0][wj];
    for(int q = 1; q < 8; q++) sum = qr_add(sum, sW[q][wi0][wj]);
    sX[wi0][wj] = sum;
    __syncthreads();
    T y = S::zero();
#pragma unroll
    for(int k = 0; k < QW; k++) y = ADJ ? S::fma_cj(sT[k][wi0], sX[k][wj], y) : S::fma_(sT[wi0][k], sX[k][wj], y);
    sW[0][wi0][wj] = y;  // read by the barrier's other side only
    __syncthreads();
    for(int r0 = 16 * w; r0 < rows; r0 += 128) {
        T a0[4], a1[4];
#pragma unroll
        for(int k = 0; k < 4; k++) a0[k] = v(r0 + g, 4 * k + t), a1[k] = v(r0 + g + 8, 4 * k + t);
#pragma unroll
        for(int q = 0; q < 2; q++) {
            double re[4] = {}, im[4] = {};
#pragma unroll
            for(int k = 0; k < 4; k++) {
                const T b = sW[0][4 * k + t][q * 8 + g];
                if constexpr(!C) {
                    dmma_f64(re, a0[k], a1[k], b);
                } else {
                    dmma_f64(re, a0[k].x, a1[k].x, b.x);
                    dmma_f64(im, a0[k].x, a1[k].x, b.y);
                    dmma_f64(re, -a0[k].y, -a1[k].y, b.y);
                    dmma_f64(im, a0[k].y, a1[k].y, b.x);
                }
            }
#pragma unroll
            for(int u = 0; u < 4; u++) {
                const int r = r0 + g + 8 * (u >> 1), c = q * 8 + 2 * t + (u & 1);
                if(r < rows && c < cw) {
                    T *p = Ap + r + lda * (int64_t)c;
                    if constexpr(!C)
                        *p -= re[u];
                    else
                        *p = make_double2(p->x - re[u], p->y - im[u]);
                }
            }
        }
    }
}

int &last_svd_sweeps() {
    static thread_local int n = 0;
    return n;
}

static int g1(int64_t n) {
    int64_t g = (n + 255) / 256, cap = (int64_t)device_sm_count() * 8;
    return (int)(g < 1 ? 1 : (g < cap ? g : cap));
}

// Rank rule of svd.cpp:257-280 on descending sigma (only exactly-nonzero values count, like
// svd_lapacke.cpp:453 S.nonZeros()).  Returns rank (>0) or -1 (the reference throws there).
int64_t truncation_rank(const double *S, int64_t n, int64_t rank_max, int64_t rank_min, double lim, double *trunc_err) {
    int64_t nz = 0;
    for(int64_t i = 0; i < n; i++) nz += S[i] != 0.0;
    std::vector<double> err(nz + 1, 0.0);
    double              acc = 0;
    for(int64_t s = nz; s >= 0; s--) {
        if(s < nz) acc += S[s] * S[s];
        err[s] = std::sqrt(acc);
    }
    int64_t rank = 0;
    for(int64_t s = 0; s <= nz; s++) rank += err[s] >= lim;
    int64_t rank_lim = nz;
    if(rank_max > 0) rank_lim = std::min(nz, rank_max);
    rank = std::min(rank, rank_lim);
    if(rank_min > 0) rank = std::max(rank, std::min(nz, rank_min));
    if(rank <= 0) return -1;
    if(trunc_err) *trunc_err = err[rank];
    return rank;
}

// Factorisations before Jacobi, for A in its tall orientation:
//   2  A P = Q1 R1, R1^H = Q2 R2, Jacobi on R2^H;   1  A = Q1 R1 (one panel), Jacobi on R1;   0  Jacobi on A.
// Both factorisations cost about 2.3 us a column and eight launches, and save sweeps, most on graded spectra; one factor alone
// makes a long matrix short enough for shared memory.  us for none / one / both, Gaussian | graded: real 16 x 16 151 / - / 195 |
// 222 / - / 230, 17 x 17 177 / - / 279 | 240 / - / 238, 32 x 32 252 / - / 317 | 490 / - / 278, 256 x 4 118 / 96 / - | 118 / 93 / -,
// 300 x 8 187 / 121 / 154 | 200 / 132 / 137, 300 x 16 255 / 170 / 195 | 400 / 241 / 170; complex 256 x 16 342 / 245 / - |
// 637 / 350 / -.  A panel of more than ROWS_MAX rows does not fit the registers of a cluster of eight CTAs.
template<class T>
static int svd_factors(int64_t M, int64_t N) {
    if(M > QrPanel<T>::ROWS_MAX) return 0;
    if(N > QW + 1 || (N > QW && M > JW_ROWS) || (N >= 10 && M > 256)) return 2;
    return M > (N == 1 ? 256 : JW_ROWS) ? 1 : 0;
}

// Scratch of one SVD, in its tall orientation (M = max, N = min of the dims): G (M x npad: A, then Q1's vectors and R1) and V
// (npad x npad); with factors Y (npad x npad: Jacobi's matrix, then the right vectors), the panels' T factors and, for a wide A, Z
// (M x npad: A^H, then the left vectors); with two also X (npad x npad: Q2's vectors); the norms and orders.
static int64_t svd_bytes(int64_t M, int64_t N, int qr, bool wide, int64_t esize) {
    const int64_t npad = (N + JP - 1) / JP * JP, ldg = (M + 1) / 2 * 2;
    return esize * (ldg * npad * (qr && wide ? 2 : 1) + npad * npad * (1 + qr) + (qr ? 2 * QW * npad : 0)) + 8 * (2 * npad + 64) + 4 * (3 * npad + 64) + 256;
}
int64_t svd_scratch_bytes(int64_t m, int64_t n, int64_t esize, bool flat) {
    const int64_t M = std::max(m, n), N = std::min(m, n);
    return svd_bytes(M, N, flat ? 0 : (esize == 16 ? svd_factors<double2>(M, N) : svd_factors<double>(M, N)), m < n, esize);
}
// Enough for every matrix of up to m rows and n columns (a workspace that serves many shapes).
int64_t svd_scratch_max(int64_t m, int64_t n, int64_t esize) {
    const int64_t M = std::max(m, n), N = std::min(m, n), Mq = std::min<int64_t>(M, esize == 16 ? QrPanel<double2>::ROWS_MAX : QrPanel<double>::ROWS_MAX);
    return std::max(svd_bytes(M, N, 0, false, esize), svd_bytes(Mq, std::min(N, Mq), 2, true, esize));
}

// In-place QR of G (M x N, leading dim ldg); the panels' T factors go to Tf (QW x QW each).
template<class T>
static int qr_factor(T *G, int64_t ldg, int M, int N, T *Tf, cudaStream_t s) {
    constexpr int RPT = QrPanel<T>::RPT;
    for(int j0 = 0; j0 < N; j0 += QW) {
        const int w = std::min(QW, N - j0), rows = M - j0;
        const int thr = rows <= QrPanel<T>::THR_MIN * RPT ? QrPanel<T>::THR_MIN : QrPanel<T>::THR_MAX;
        int       CL  = 1;
        while(CL * RPT * thr < rows) CL *= 2;
        T *Tp = Tf + (int64_t)(j0 / QW) * QW * QW;
        HEFF_CUDA((launch_chained_cluster((unsigned)CL, qr_panel_kernel<T>, CL, thr + 32, 0, s, G, ldg, M, j0, w, Tp, CL)));
        const int rest = N - j0 - w;
        if(rest > 0) {
            HEFF_CUDA((launch_chained(qr_apply_kernel<T, true>, (rest + QW - 1) / QW, 256, 0, s, G, ldg, M, j0, Tp, G + ldg * (int64_t)(j0 + w), ldg, rest)));
        }
    }
    return HEFF_OK;
}
// A (M x nc) <- Q A for the factors that qr_factor left in G (N columns)
template<class T>
static int qr_apply_q(const T *G, int64_t ldg, int M, int N, const T *Tf, T *A, int64_t lda, int nc, cudaStream_t s) {
    for(int j0 = (N - 1) / QW * QW; j0 >= 0; j0 -= QW) {
        HEFF_CUDA((launch_chained(qr_apply_kernel<T, false>, (nc + QW - 1) / QW, 256, 0, s, G, ldg, M, j0, Tf + (int64_t)(j0 / QW) * QW * QW, A, lda, nc)));
    }
    return HEFF_OK;
}

// Shared-memory opt-in of the Jacobi kernels, once per device.
template<class T>
static int jacobi_attributes() {
    static int done[64] = {0};
    int        dev      = 0;
    HEFF_CUDA(cudaGetDevice(&dev));
    if(dev < 0 || dev >= 64 || !done[dev]) {
        HEFF_CUDA(cudaFuncSetAttribute(jacobi_round_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jacobi_round_bytes<T>()));
        HEFF_CUDA(cudaFuncSetAttribute(jacobi_whole_kernel<T, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jacobi_whole_bytes<T, 32>()));
        HEFF_CUDA(cudaFuncSetAttribute(jacobi_whole_kernel<T, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jacobi_whole_bytes<T, 64>()));
        if(dev >= 0 && dev < 64) done[dev] = 1;
    }
    return HEFF_OK;
}

// Full SVD driver.  A: m x n (lda), not modified.  Outputs (device): U (m x kmax), S (kmax), VT (kmax x n)
// with kmax = min(m, n, rank_max>0 ? rank_max : inf); *rank and *trunc_err on the host.  flat: the caller knows that the
// singular values lie close together, so factors would save no sweeps.
template<class T>
static int svd_truncated_t(const T *A, int64_t lda, int64_t m, int64_t n, int64_t rank_max, double trunc_lim, T *U, double *S, T *VT, int64_t *rank,
                           double *trunc_err, void *scratch, int *sweeps_out, cudaStream_t s, bool flat = false) {
    if(m <= 0 || n <= 0 || m > (1 << 24) || n > 16384) return HEFF_BAD_SHAPE;
    HEFF_TRY(jacobi_attributes<T>());
    const bool    wide = m < n;  // worked on as A^H
    const int     M = (int)std::max(m, n), N = (int)std::min(m, n);
    const int     npad = (N + JP - 1) / JP * JP;
    const int64_t ldg  = (M + 1) / 2 * 2;
    const int     qr   = flat ? 0 : svd_factors<T>(M, N);
    const bool    precond = qr > 0;
    T            *G    = reinterpret_cast<T *>(scratch);
    T            *Z    = G + ldg * npad;
    T            *V    = Z + (precond && wide ? ldg * npad : 0);
    T            *Y    = V + (int64_t)npad * npad;
    T            *X    = Y + (precond ? (int64_t)npad * npad : 0);
    T            *T1 = X + (qr == 2 ? (int64_t)npad * npad : 0), *T2 = T1 + (precond ? QW * npad : 0);
    double       *sig  = reinterpret_cast<double *>(T2 + (precond ? QW * npad : 0));  // column norms
    double       *dmax = sig + npad;  // [0] largest squared column norm of a sweep; [1] (int) pairs rotated in it, or sweeps run
    int          *drot = reinterpret_cast<int *>(dmax + 1);
    double       *sig0 = dmax + 64;   // norms of A's columns
    int          *perm = reinterpret_cast<int *>(sig0 + npad);
    int          *cmap = perm + npad;  // column order of the current sweep (block b = columns cmap[16 b .. 16 b + 15])
    int          *cord = cmap + npad;  // order of A's columns in G
    auto norms_order = [&](const T *W, int64_t ldw, int rows, int cols, double *nrm, int *ord) -> int {
        HEFF_CUDA((launch_chained(col_norms_kernel<T>, (cols * 32 + 255) / 256, 256, 0, s, W, ldw, rows, cols, nrm)));
        HEFF_CUDA((launch_chained(col_order_kernel, (cols + 127) / 128, 128, 0, s, nrm, cols, ord)));
        return HEFF_OK;
    };
    T            *W    = precond ? Y : G;  // the matrix Jacobi works on, rows x npad
    const int64_t ldw  = precond ? npad : ldg;
    const int     rows = precond ? N : M;
    const bool    whole = npad <= JW_P && rows <= 1024;
    const T      *src  = A;
    int64_t       lds  = lda;
    if(wide && (precond || !whole)) {
        T *dst = qr == 2 ? Z : G;
        HEFF_CUDA(cudaMemsetAsync(dst, 0, sizeof(T) * (size_t)ldg * (qr == 1 ? QW : npad), s));  // a panel is read in whole
        HEFF_CUDA((launch_chained(adjoint_kernel<T, false>, dim3((unsigned)cdiv(N, 32), (unsigned)cdiv(M, 32)), 256, 0, s, A, lda, (int)m, (int)n, dst, ldg, M, N)));
        src = dst, lds = ldg;
    }
    const dim3 sq((unsigned)(npad / 32), (unsigned)(npad / 32));
    if(qr == 2) {
        // G = A or A^H with the columns by descending norm: the factors of a matrix whose columns differ by orders of
        // magnitude keep each column's own relative accuracy, and zero columns come last
        HEFF_TRY(norms_order(src, lds, M, N, sig0, cord));
        HEFF_CUDA((launch_chained(copy_pad_kernel<T>, g1(ldg * npad), 256, 0, s, src, lds, M, N, G, ldg, npad, cord)));
        HEFF_TRY(qr_factor<T>(G, ldg, M, N, T1, s));
        HEFF_CUDA((launch_chained(adjoint_kernel<T, true>, sq, 256, 0, s, G, ldg, N, N, X, npad, npad, npad)));
        HEFF_TRY(qr_factor<T>(X, npad, N, N, T2, s));
        HEFF_CUDA((launch_chained(adjoint_kernel<T, true>, sq, 256, 0, s, X, npad, N, N, Y, npad, npad, npad)));
    } else if(qr == 1) {  // a zero column stays exactly zero through the factorisation
        if(!wide) HEFF_CUDA((launch_chained(copy_pad_kernel<T>, g1(ldg * QW), 256, 0, s, src, lds, M, N, G, ldg, QW, nullptr)));
        HEFF_TRY(qr_factor<T>(G, ldg, M, N, T1, s));
        HEFF_CUDA((launch_chained(adjoint_kernel<T, true>, sq, 256, 0, s, G, ldg, N, N, Y, npad, npad, npad)));  // R1^H
    } else if(!wide && !whole) {
        HEFF_CUDA((launch_chained(copy_pad_kernel<T>, g1(ldg * npad), 256, 0, s, src, lds, M, N, G, ldg, npad, nullptr)));
    }
    const int B = npad / JB;  // even
    // off-diagonal tolerance just above the rounding noise of a length-m dot product
    const double        tol   = std::max(1e-14, 8.0 * 2.2e-16 * std::sqrt((double)M));
    const double        eps   = 2.220446049250313e-16;
    int                 sweep = 0;
    std::vector<double> host(2 * npad + 64);  // sig | dmax | sig0
    if(whole) {
        const T      *from = precond ? W : A;
        const int64_t ldf  = precond ? ldw : lda;
        const int     adj  = qr == 1 || (!precond && wide);
        if(npad == 32)
            HEFF_CUDA((launch_chained(jacobi_whole_kernel<T, 32>, 1, jw_thr(32), jacobi_whole_bytes<T, 32>(), s, from, ldf, adj, W, ldw, rows, N, V, tol, JOUTER, sig, drot)));
        else
            HEFF_CUDA((launch_chained(jacobi_whole_kernel<T, 64>, 1, jw_thr(64), jacobi_whole_bytes<T, 64>(), s, from, ldf, adj, W, ldw, rows, N, V, tol, JOUTER, sig, drot)));
    } else {
        HEFF_CUDA((launch_chained(eye_kernel<T>, g1((int64_t)npad * npad), 256, 0, s, V, npad, npad)));
        // Norm-ordered blocks (the block form of de Rijk's pivoting in LAPACK's ?gesvj): before every sweep the
        // columns are ordered by norm and blocks are formed from neighbours, so clusters of close singular values
        // meet inside one pair block.  CTAs per pair: enough to fill the SMs with one wave (the pairs of a round are only
        // B / 2), when the rows are long enough to share out.
        int CL = 1;
        while(CL < JCL && (int64_t)(B / 2) * CL * 2 <= device_sm_count() && rows >= 64 * CL * 2) CL *= 2;
        double floor_abs = 0.0;  // first sweep: relative criterion only
        for(; sweep < JOUTER; sweep++) {
            HEFF_TRY(norms_order(W, ldw, rows, npad, sig, cmap));
            HEFF_CUDA(cudaMemsetAsync(dmax, 0, 2 * sizeof(double), s));
            for(int r = 0; r < B - 1; r++) {
                HEFF_CUDA((launch_chained_cluster((unsigned)CL, jacobi_round_kernel<T>, B / 2 * CL, JTHR, jacobi_round_bytes<T>(), s, W, ldw, rows, V, npad,
                                                  npad, B, r, tol, floor_abs, cmap, dmax, drot, CL)));
            }
            struct {
                double gmax;
                int    rot;
            } st{};
            HEFF_CUDA(cudaMemcpyAsync(&st, dmax, sizeof(st), cudaMemcpyDeviceToHost, s));
            HEFF_CUDA(cudaStreamSynchronize(s));
            if(st.rot == 0) break;
            floor_abs = (double)rows * eps * eps * st.gmax;
        }
        HEFF_CUDA((launch_chained(col_norms_kernel<T>, (npad * 32 + 255) / 256, 256, 0, s, W, ldw, rows, npad, sig)));
    }
    HEFF_CUDA(cudaMemcpyAsync(host.data(), sig, sizeof(double) * host.size(), cudaMemcpyDeviceToHost, s));
    HEFF_CUDA(cudaStreamSynchronize(s));
    if(whole) {
        int ran = 0;
        std::memcpy(&ran, &host[npad + 1], sizeof(int));
        sweep = ran - 1;
    }
    last_svd_sweeps() = sweep + 1;
    if(sweeps_out) *sweeps_out = sweep + 1;
    std::vector<int> order(npad);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return host[a] > host[b]; });
    std::vector<double> sorted(N);
    for(int i = 0; i < N; i++) sorted[i] = host[order[i]];
    if(qr == 2) {  // as many zero singular values as zero columns (the factorisation leaves rounding noise in their place)
        int nzero = 0;
        for(int i = 0; i < N; i++) nzero += host[npad + 64 + i] == 0.0;
        for(int i = 0; i < nzero; i++) sorted[N - 1 - i] = 0.0;
    }
    const int64_t r = truncation_rank(sorted.data(), N, rank_max, 0, trunc_lim, trunc_err);
    if(r <= 0) {
        set_last_error_msg("svd: rank <= 0 (all singular values zero or below the truncation limit)");
        return HEFF_BAD_ARG;
    }
    *rank = r;
    HEFF_CUDA(cudaMemcpyAsync(perm, order.data(), sizeof(int) * r, cudaMemcpyHostToDevice, s));
    // ---- singular vectors: left = Q1 [U_j; 0] (M x r), right = P Q2 V_j or V_j (N x r); U and VT, exchanged for a wide A
    const int kk = (int)r, gr = g1((int64_t)(M + N) * r);
    if(!precond) {
        if(!wide)
            HEFF_CUDA((launch_chained(take_columns_kernel<T, false, true>, gr, 256, 0, s, W, ldw, rows, V, npad, N, perm, sig, kk, S, U, M, M, VT, 0)));
        else
            HEFF_CUDA((launch_chained(take_columns_kernel<T, true, false>, gr, 256, 0, s, W, ldw, rows, V, npad, N, perm, sig, kk, S, VT, 0, M, U, N)));
    } else if(qr == 1) {
        T            *left = wide ? Z : U;
        const int64_t ldl  = wide ? ldg : M;
        if(!wide)
            HEFF_CUDA((launch_chained(take_columns_kernel<T, false, true>, gr, 256, 0, s, W, ldw, rows, V, npad, N, perm, sig, kk, S, left, ldl, M, VT, 0)));
        else
            HEFF_CUDA((launch_chained(take_columns_kernel<T, false, false>, gr, 256, 0, s, W, ldw, rows, V, npad, N, perm, sig, kk, S, left, ldl, M, U, N)));
        HEFF_TRY(qr_apply_q<T>(G, ldg, M, N, T1, left, ldl, kk, s));
        if(wide) HEFF_CUDA((launch_chained(adjoint_rows_kernel<T>, g1((int64_t)M * r), 256, 0, s, left, ldl, M, kk, nullptr, VT)));
    } else {
        T            *left = wide ? Z : U;
        const int64_t ldl  = wide ? ldg : M;
        // the right vectors take the place of the columns that the left ones come from
        T *R = Y;
        HEFF_CUDA((launch_chained(take_columns_kernel<T, false, false>, g1((int64_t)M * r), 256, 0, s, W, ldw, rows, V, npad, 0, perm, sig, kk, S, left, ldl, M, R, npad)));
        HEFF_CUDA((launch_chained(take_columns_kernel<T, false, false>, g1((int64_t)N * r), 256, 0, s, W, ldw, rows, V, npad, N, perm, sig, kk, S, left, ldl, 0, R, npad)));
        HEFF_TRY(qr_apply_q<T>(G, ldg, M, N, T1, left, ldl, kk, s));
        HEFF_TRY(qr_apply_q<T>(X, npad, N, N, T2, R, npad, kk, s));
        if(!wide) {
            HEFF_CUDA((launch_chained(adjoint_rows_kernel<T>, g1((int64_t)N * r), 256, 0, s, R, npad, N, kk, cord, VT)));
        } else {  // A^H = left S right^H: U = right, VT = left^H
            HEFF_CUDA((launch_chained(scatter_rows_kernel<T>, g1((int64_t)N * r), 256, 0, s, R, npad, N, kk, cord, U, m)));
            HEFF_CUDA((launch_chained(adjoint_rows_kernel<T>, g1((int64_t)M * r), 256, 0, s, left, ldl, M, kk, nullptr, VT)));
        }
        HEFF_LAUNCH_CHECK();
    }
    HEFF_CUDA(cudaStreamSynchronize(s));  // host vectors above must outlive the copies
    return HEFF_OK;
}

int svd_truncated(const double *A, int64_t lda, int64_t m, int64_t n, int64_t rank_max, double trunc_lim, double *U, double *S, double *VT,
                  int64_t *rank, double *trunc_err, void *scratch, int *sweeps_out, cudaStream_t s, bool flat) {
    return svd_truncated_t<double>(A, lda, m, n, rank_max, trunc_lim, U, S, VT, rank, trunc_err, scratch, sweeps_out, s, flat);
}
int svd_truncated(const double2 *A, int64_t lda, int64_t m, int64_t n, int64_t rank_max, double trunc_lim, double2 *U, double *S, double2 *VT,
                  int64_t *rank, double *trunc_err, void *scratch, int *sweeps_out, cudaStream_t s, bool flat) {
    return svd_truncated_t<double2>(A, lda, m, n, rank_max, trunc_lim, U, S, VT, rank, trunc_err, scratch, sweeps_out, s, flat);
}

// theta [dL*dR, chiL, chiR] -> A[(s1 + dL a), (s2 + dR b)] = theta[s1 + dL s2, a, b]   (svd.h:217 reshape+shuffle)
template<class T>
__global__ void schmidt_pack_kernel(const T *__restrict__ th, T *__restrict__ A, int64_t dL, int64_t dR, int64_t cL, int64_t cR) {
    grid_wait();
    const int64_t m = dL * cL, tot = m * dR * cR;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = e % m, col = e / m;
        const int64_t s1 = row % dL, a = row / dL, s2 = col % dR, b = col / dR;
        A[e]             = th[(s1 + dL * s2) + dL * dR * (a + cL * b)];
    }
}
// VT [k, dR*chiR] -> V [dR, k, chiR] (svd.h:173 shuffle {1,0,2});  S <- S / ||S||
template<class T>
__global__ void schmidt_unpack_kernel(const T *__restrict__ VT, T *__restrict__ Vout, double *__restrict__ S, double inv_norm, int64_t k, int64_t dR,
                                      int64_t cR) {
    grid_wait();
    const int64_t tot = k * dR * cR;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s2 = e % dR, r = e / dR, i = r % k, b = r / k;
        Vout[e]          = VT[i + k * (s2 + dR * b)];
        if(e < k) S[e] *= inv_norm;
    }
}

// for the split of one theta, and of every theta of up to these bonds
static int64_t schmidt_bytes(int64_t m, int64_t n, int64_t rank_max, int64_t svd, int64_t esize) {
    const int64_t kmax = std::min(std::min(m, n), rank_max > 0 ? rank_max : INT64_MAX);
    return esize * ((m * n + 31) / 32 * 32 + (kmax * n + 31) / 32 * 32) + svd + 512;
}
int64_t schmidt_scratch_bytes(int64_t dL, int64_t dR, int64_t cL, int64_t cR, int64_t rank_max, int64_t esize) {
    return schmidt_bytes(dL * cL, dR * cR, rank_max, svd_scratch_bytes(dL * cL, dR * cR, esize), esize);
}
int64_t schmidt_scratch_max(int64_t dL, int64_t dR, int64_t cL, int64_t cR, int64_t rank_max, int64_t esize) {
    return schmidt_bytes(dL * cL, dR * cR, rank_max, svd_scratch_max(dL * cL, dR * cR, esize), esize);
}

template<class T>
static int schmidt_split_t(const T *theta, int64_t dL, int64_t dR, int64_t cL, int64_t cR, int64_t rank_max, double trunc_lim, T *U, double *S, T *V,
                           int64_t *rank, double *trunc_err, void *scratch, cudaStream_t s) {
    const int64_t m = dL * cL, n = dR * cR;
    T            *A    = reinterpret_cast<T *>(scratch);
    T            *VT   = A + (m * n + 31) / 32 * 32;
    const int64_t kmax = std::min(std::min(m, n), rank_max > 0 ? rank_max : INT64_MAX);
    void         *jscr = VT + (kmax * n + 31) / 32 * 32;
    HEFF_CUDA((launch_chained(schmidt_pack_kernel<T>, g1(m * n), 256, 0, s, theta, A, dL, dR, cL, cR)));
    HEFF_TRY(svd_truncated_t<T>(A, m, m, n, rank_max, trunc_lim, U, S, VT, rank, trunc_err, jscr, nullptr, s));
    std::vector<double> hs(*rank);
    HEFF_CUDA(cudaMemcpyAsync(hs.data(), S, sizeof(double) * (*rank), cudaMemcpyDeviceToHost, s));
    HEFF_CUDA(cudaStreamSynchronize(s));
    double nrm = 0;
    for(double v : hs) nrm += v * v;
    nrm = std::sqrt(nrm);
    HEFF_CUDA((launch_chained(schmidt_unpack_kernel<T>, g1((*rank) * n), 256, 0, s, VT, V, S, nrm > 0 ? 1.0 / nrm : 1.0, *rank, dR, cR)));
    return HEFF_OK;
}

int schmidt_split(const double *theta, int64_t dL, int64_t dR, int64_t cL, int64_t cR, int64_t rank_max, double trunc_lim, double *U, double *S,
                  double *V, int64_t *rank, double *trunc_err, void *scratch, cudaStream_t s) {
    return schmidt_split_t<double>(theta, dL, dR, cL, cR, rank_max, trunc_lim, U, S, V, rank, trunc_err, scratch, s);
}
int schmidt_split(const double2 *theta, int64_t dL, int64_t dR, int64_t cL, int64_t cR, int64_t rank_max, double trunc_lim, double2 *U, double *S,
                  double2 *V, int64_t *rank, double *trunc_err, void *scratch, cudaStream_t s) {
    return schmidt_split_t<double2>(theta, dL, dR, cL, cR, rank_max, trunc_lim, U, S, V, rank, trunc_err, scratch, s);
}

}  // namespace heff

using namespace heff;

template<class T>
static int svd_entry(const T *A, int64_t rows, int64_t cols, int64_t rank_max, double trunc_lim, T *U, double *S, T *VT, int64_t *rank,
                     double *trunc_err, void *stream) {
    if(!A || !U || !S || !VT || !rank || rows <= 0 || cols <= 0) return HEFF_BAD_ARG;
    cudaStream_t s    = (cudaStream_t)stream;
    void        *base = nullptr;
    HEFF_TRY(stream_workspace(s, (size_t)svd_scratch_bytes(rows, cols, sizeof(T)), &base));
    double te = 0;
    HEFF_TRY(svd_truncated(A, rows, rows, cols, rank_max, trunc_lim, U, S, VT, rank, &te, base, nullptr, s));
    if(trunc_err) *trunc_err = te;
    return HEFF_OK;
}

template<class T>
static int schmidt_entry(const T *theta, int64_t dL, int64_t dR, int64_t chiL, int64_t chiR, int64_t rank_max, double trunc_lim, T *U, double *S, T *V,
                         int64_t *rank, double *trunc_err, void *stream) {
    if(!theta || !U || !S || !V || !rank || dL <= 0 || dR <= 0 || chiL <= 0 || chiR <= 0) return HEFF_BAD_ARG;
    cudaStream_t s    = (cudaStream_t)stream;
    void        *base = nullptr;
    HEFF_TRY(stream_workspace(s, (size_t)schmidt_scratch_bytes(dL, dR, chiL, chiR, rank_max, sizeof(T)), &base));
    double te = 0;
    HEFF_TRY(schmidt_split(theta, dL, dR, chiL, chiR, rank_max, trunc_lim, U, S, V, rank, &te, base, s));
    if(trunc_err) *trunc_err = te;
    return HEFF_OK;
}

extern "C" int heff_svd_d(const double *A, int64_t rows, int64_t cols, int64_t rank_max, double trunc_lim, double *U, double *S, double *VT,
                          int64_t *rank, double *trunc_err, void *stream) {
    return svd_entry<double>(A, rows, cols, rank_max, trunc_lim, U, S, VT, rank, trunc_err, stream);
}

extern "C" int heff_svd_z(const heff_z *A, int64_t rows, int64_t cols, int64_t rank_max, double trunc_lim, heff_z *U, double *S, heff_z *VT,
                          int64_t *rank, double *trunc_err, void *stream) {
    return svd_entry<double2>(reinterpret_cast<const double2 *>(A), rows, cols, rank_max, trunc_lim, reinterpret_cast<double2 *>(U), S,
                              reinterpret_cast<double2 *>(VT), rank, trunc_err, stream);
}

extern "C" int heff_schmidt_d(const double *theta, int64_t dL, int64_t dR, int64_t chiL, int64_t chiR, int64_t rank_max, double trunc_lim, double *U,
                              double *S, double *V, int64_t *rank, double *trunc_err, void *stream) {
    return schmidt_entry<double>(theta, dL, dR, chiL, chiR, rank_max, trunc_lim, U, S, V, rank, trunc_err, stream);
}

extern "C" int heff_schmidt_z(const heff_z *theta, int64_t dL, int64_t dR, int64_t chiL, int64_t chiR, int64_t rank_max, double trunc_lim, heff_z *U,
                              double *S, heff_z *V, int64_t *rank, double *trunc_err, void *stream) {
    return schmidt_entry<double2>(reinterpret_cast<const double2 *>(theta), dL, dR, chiL, chiR, rank_max, trunc_lim, reinterpret_cast<double2 *>(U), S,
                                  reinterpret_cast<double2 *>(V), rank, trunc_err, stream);
}
