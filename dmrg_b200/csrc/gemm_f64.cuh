// FP64 / complex128 batched GEMM on the sm_100a FP64 tensor pipe (DMMA, mma.sync.m16n8k4.f64).
//
// tcgen05.mma has no f64 kind, so the FP64 tensor path on Blackwell is the warp-level DMMA instruction: 64 FMAs
// per clock and SM (36.9 TFLOP/s at 1.95 GHz, measured with register operands; m16n8k8 and m16n8k16 run at the
// same rate).  Operands are staged global -> shared through a multistage cp.async pipeline (16-byte copies where the
// layout allows, zero-fill at the edges); padded shared tiles make every fragment load bank-conflict free.
//
//   C[b] = alpha * op(A[b]) * op(B[b]) + beta * C[b]      (column-major, BLAS conventions)
//   op(A) = A (M x K, m contiguous)   or  A^T (A stored K x M, k contiguous)   [TA]
//   op(B) = B (K x N, k contiguous)   or  B^T (B stored N x K, n contiguous)   [TB]
//   complex: 3 real DMMAs per fragment pair (3M / Gauss): t1 = ar br, t2 = ai bi, t3 = (ar + ai)(br + bi)
//   accumulated over K, then Re = t1 - t2, Im = t3 - t1 - t2 (normwise error a small constant times the 4M
//   product's, eps sqrt(K) |A| |B|).
#pragma once
#include "heff_common.cuh"

namespace heff {

struct GemmArgs {
    int         M, N, K, batch;
    const void *A;
    int64_t     lda, sA;
    const void *B;
    int64_t     ldb, sB;
    void       *C;
    int64_t     ldc, sC;
    double2     alpha, beta;  // real GEMMs use .x
    // Optional scratch for the tail split (set by the caller; nullptr or too small: no tail split).  When the
    // tiles do not fill whole waves of the device, the tiles of the last partial wave are split along K
    // into `split` pieces that write partial tiles to `part`; a second kernel sums the pieces in piece
    // order (deterministic) and applies alpha/beta.  Set by the launcher: split, nfull, part.
    void       *split_ws;
    size_t      split_ws_bytes;
    int         split, nfull;
    void       *part;
    // Set by the launcher: K pieces of every tile, one CTA of a cluster each (1 = none; then split == 1), and the
    // number of work units (whole tiles, tail pieces or cluster pieces, all batch members).
    int         cluster, units;
};

// Tile shapes.  0: large products, one CTA per SM.  1 and 2: products whose large tiles would leave SMs idle --
// the DMMA rate of an SM is the same for any tile, so a product with few tiles is as fast as the number of SMs it
// reaches (chosen by gemm_pick in gemm_f64.cu).
template<bool CPLX, int CFG>
struct GemmTile;
template<int BM_, int BN_, int BK_, int WM_, int WN_, int ST_, int MINB_, int PAD_MN_, int PAD_K_>
struct GemmTileDef {
    static constexpr int BM = BM_, BN = BN_, BK = BK_, WM = WM_, WN = WN_, STAGES = ST_, MINB = MINB_;
    static constexpr int THREADS = 32 * (BM / WM) * (BN / WN);
    static constexpr int PAD_MN = PAD_MN_, PAD_K = PAD_K_;
};
// real: a leading dim == 4 (mod 16) doubles makes the 8-byte fragment loads conflict-free
template<>
struct GemmTile<false, 0> : GemmTileDef<128, 128, 32, 64, 32, 3, 1, 4, 4> {};
template<>
struct GemmTile<false, 1> : GemmTileDef<64, 64, 32, 32, 16, 4, 1, 4, 4> {};
template<>
struct GemmTile<false, 2> : GemmTileDef<32, 32, 32, 16, 16, 4, 3, 4, 4> {};
// complex: a leading dim == 2 (mod 8) elements (m/n-major tile) or 4 (mod 8) (k-major) for the 16-byte loads
template<>
struct GemmTile<true, 0> : GemmTileDef<64, 64, 32, 32, 16, 3, 1, 2, 4> {};
template<>
struct GemmTile<true, 1> : GemmTileDef<32, 32, 32, 16, 16, 3, 2, 2, 4> {};
constexpr int gemm_cfgs(bool cplx) { return cplx ? 2 : 3; }

template<bool CPLX, int CFG, bool TA, bool TB>
struct GemmSmem {
    using G                  = GemmTile<CPLX, CFG>;
    using T                  = typename Scalar<CPLX>::T;
    static constexpr int LDA = TA ? (G::BK + G::PAD_K) : (G::BM + G::PAD_MN);  // row length of the A tile
    static constexpr int LDB = TB ? (G::BN + G::PAD_MN) : (G::BK + G::PAD_K);
    static constexpr int A_ELEMS = TA ? G::BM * LDA : G::BK * LDA;
    static constexpr int B_ELEMS = TB ? G::BK * LDB : G::BN * LDB;
    static constexpr int STAGE   = A_ELEMS + B_ELEMS;
    static constexpr size_t BYTES = (size_t)STAGE * G::STAGES * sizeof(T);
    static_assert(BYTES >= (size_t)G::BM * G::BN * sizeof(T), "the cluster reduction reuses the stages for one tile");
};

constexpr int GROUP_M = 16;  // row panels per rasterisation group

// Grouped rasterisation: consecutive tile ids walk GROUP_M row panels for every column panel, so the
// CTAs resident at one time share their A and B panels in L2 instead of re-reading them from HBM.
template<int BM, int BN>
__device__ __forceinline__ void gemm_raster(int pid, int M, int N, int &tile_m, int &tile_n) {
    const int num_m = (M + BM - 1) / BM, num_n = (N + BN - 1) / BN;
    const int per_group = GROUP_M * num_n;
    const int first_m   = (pid / per_group) * GROUP_M;
    const int gsize     = min(num_m - first_m, GROUP_M);
    tile_m              = first_m + (pid % per_group) % gsize;
    tile_n              = (pid % per_group) / gsize;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

template<int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, bool valid) {
    const int n = valid ? BYTES : 0;  // src-size 0 -> destination is zero-filled, nothing is read
    if constexpr(BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template<int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a0), "d"(a1), "d"(b0));
}

// One operand's copies of a k-tile by one thread: N chunks of EPC elements, chunk i STEP rows (k-major tile, KM) or
// STEP k's (m/n-major tile) after chunk 0, so a chunk's address is one base pointer plus a constant multiple of a
// stride kept in registers.  The pointer arithmetic of the previous form (a division, two 64-bit multiplies and the
// edge tests per chunk, all issued between the barrier and the first MMA) kept the tensor pipe idle ~7 % of the time.
template<class G, class T, bool KM, int ROWS, int EPC, int LD>
struct TileLoader {
    static constexpr int CPR  = (KM ? G::BK : ROWS) / EPC;
    static constexpr int STEP = G::THREADS / CPR;
    static constexpr int N    = ROWS * G::BK / EPC / G::THREADS;
    static_assert(G::THREADS % CPR == 0 && N >= 1 && N * STEP == (KM ? ROWS : G::BK), "chunks tile the operand");
    const T *base, *g;
    int64_t  step, next;
    int      fix, var0, row_lim;
    uint32_t dst;
    __device__ __forceinline__ void init(int tid) {
        fix  = (tid % CPR) * EPC;
        var0 = tid / CPR;
        dst  = (uint32_t)((var0 * LD + fix) * sizeof(T));
    }
    // rows r0 .. of an operand with `rows` rows, k from k0
    __device__ __forceinline__ void unit(const T *b, int64_t ld, int r0, int rows, int k0) {
        base    = b;
        g       = KM ? b + (k0 + fix) + (int64_t)(r0 + var0) * ld : b + (r0 + fix) + (int64_t)(k0 + var0) * ld;
        step    = STEP * ld;
        next    = KM ? (int64_t)G::BK : G::BK * ld;
        row_lim = rows - r0;
    }
    __device__ __forceinline__ void copy(int i, uint32_t stage, int k_lim) const {
        const bool v = KM ? (var0 + i * STEP < row_lim && fix < k_lim) : (fix < row_lim && var0 + i * STEP < k_lim);
        cp_async<EPC * (int)sizeof(T)>(stage + dst + (uint32_t)(i * STEP * LD * sizeof(T)), v ? g + i * step : base, v);
    }
};

// Work unit u of a GEMM: a whole tile, a K piece of a tail tile (tail split) or of any tile (cluster split).
struct GemmUnit {
    int tile, bz, kt0, kt1, piece;  // piece >= 0: index of the partial tile of a tail piece
};
__device__ __forceinline__ GemmUnit gemm_unit(const GemmArgs &p, int u, int tiles, int KT) {
    GemmUnit w{u, 0, 0, KT, -1};
    if(p.cluster > 1) {
        const int q = u % p.cluster;
        w.tile      = u / p.cluster;
        w.kt0       = (int)((int64_t)KT * q / p.cluster);
        w.kt1       = (int)((int64_t)KT * (q + 1) / p.cluster);
    } else if(p.split > 1 && u >= p.nfull) {
        w.piece     = u - p.nfull;
        const int q = w.piece % p.split;
        w.tile      = p.nfull + w.piece / p.split;
        w.kt0       = (int)((int64_t)KT * q / p.split);
        w.kt1       = (int)((int64_t)KT * (q + 1) / p.split);
    }
    w.bz   = w.tile / tiles;
    w.tile = w.tile % tiles;
    return w;
}

// Persistent GEMM: each CTA walks the work units blockIdx.x, + gridDim.x, ... as one stream of k-tiles.  The copies
// run STAGES - 1 k-tiles ahead across unit boundaries (a unit's first tiles load during the previous unit's last
// k-steps and epilogue) and are spread over the k-steps; the next k-step's fragments load while the current one's
// MMAs issue, so the tensor pipe waits neither for shared memory nor at the k-tile barrier.  VEC = elements per
// cp.async (2 doubles or 1).
template<bool CPLX, int CFG, bool TA, bool TB, int VEC>
__global__ void __launch_bounds__(GemmTile<CPLX, CFG>::THREADS, GemmTile<CPLX, CFG>::MINB) gemm_f64_kernel(const GemmArgs p) {
    grid_wait();
    using G  = GemmTile<CPLX, CFG>;
    using SM = GemmSmem<CPLX, CFG, TA, TB>;
    using T  = typename Scalar<CPLX>::T;
    constexpr int BM = G::BM, BN = G::BN, BK = G::BK, WM = G::WM, WN = G::WN, ST = G::STAGES, THR = G::THREADS;
    constexpr int MT = WM / 16, NT = WN / 8, NK = BK / 4;  // mma tiles per warp, k-steps per k-tile
    constexpr int EPC = CPLX ? 1 : VEC;                    // elements per copy
    using LA = TileLoader<G, T, TA, BM, EPC, SM::LDA>;
    using LB = TileLoader<G, T, !TB, BN, EPC, SM::LDB>;
    constexpr int NCOPY = LA::N + LB::N;
    static_assert(NK % 2 == 0 && NK >= 2, "fragment buffers alternate by k-step");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T             *smem  = reinterpret_cast<T *>(smem_raw);
    const uint32_t smem0 = smem_u32(smem_raw);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm0 = (warp % (BM / WM)) * WM, wn0 = (warp / (BM / WM)) * WN;
    const int M = p.M, N = p.N, K = p.K;
    const int KT = (K + BK - 1) / BK, tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);

    // ---- the loading side of the stream: unit lu, k-tile lk of [lk, lk1)
    LA  la;
    LB  lb;
    int lu = (int)blockIdx.x, lk = 0, lk1 = 0;
    la.init(tid);
    lb.init(tid);
    auto load_unit = [&]() {
        const GemmUnit w = gemm_unit(p, lu, tiles, KT);
        int            tm, tn;
        gemm_raster<BM, BN>(w.tile, M, N, tm, tn);
        lk  = w.kt0;
        lk1 = w.kt1;
        la.unit(reinterpret_cast<const T *>(p.A) + (int64_t)w.bz * p.sA, p.lda, tm * BM, M, lk * BK);
        lb.unit(reinterpret_cast<const T *>(p.B) + (int64_t)w.bz * p.sB, p.ldb, tn * BN, N, lk * BK);
    };
    auto load_copy = [&](int q, int slot) {  // copy q of the current k-tile
        const uint32_t st = smem0 + (uint32_t)(slot * SM::STAGE * sizeof(T));
        if(q < LA::N)
            la.copy(q, st, K - lk * BK);
        else
            lb.copy(q - LA::N, st + (uint32_t)(SM::A_ELEMS * sizeof(T)), K - lk * BK);
    };
    auto load_next = [&]() {
        la.g += la.next;
        lb.g += lb.next;
        if(++lk == lk1) {
            lu += (int)gridDim.x;
            if(lu < p.units) load_unit();
        }
    };

    // ---- fragments of one k-step
    T    fa[2][MT][2], fb[2][NT];
    auto load_frag = [&](int f, int slot, int k4) {
        const T *As = smem + slot * SM::STAGE;
        const T *Bs = As + SM::A_ELEMS;
#pragma unroll
        for(int i = 0; i < MT; i++) {
            const int mr = wm0 + i * 16 + g;
            if constexpr(TA) {
                fa[f][i][0] = As[mr * SM::LDA + k4 + t];
                fa[f][i][1] = As[(mr + 8) * SM::LDA + k4 + t];
            } else {
                fa[f][i][0] = As[(k4 + t) * SM::LDA + mr];
                fa[f][i][1] = As[(k4 + t) * SM::LDA + mr + 8];
            }
        }
#pragma unroll
        for(int j = 0; j < NT; j++) {
            const int nc = wn0 + j * 8 + g;
            fb[f][j]     = TB ? Bs[(k4 + t) * SM::LDB + nc] : Bs[nc * SM::LDB + k4 + t];
        }
    };

    if(lu >= p.units) return;  // never in a cluster launch (its grid is exactly the units)
    load_unit();
#pragma unroll
    for(int s = 0; s < ST - 1; s++) {
        if(lu < p.units) {
#pragma unroll
            for(int q = 0; q < NCOPY; q++) load_copy(q, s);
            load_next();
        }
        cp_async_commit();
    }
    int slot_w = ST - 1, slot_r = 0;
    cp_async_wait<ST - 2>();
    __syncthreads();
    load_frag(0, 0, 0);

    for(int u = (int)blockIdx.x; u < p.units; u += (int)gridDim.x) {
        const GemmUnit w = gemm_unit(p, u, tiles, KT);
        double         acc[MT][NT][CPLX ? 3 : 1][4];  // complex: t1, t2, t3 of the 3M product
#pragma unroll
        for(int i = 0; i < MT; i++)
#pragma unroll
            for(int j = 0; j < NT; j++)
#pragma unroll
                for(int c = 0; c < (CPLX ? 3 : 1); c++)
#pragma unroll
                    for(int r = 0; r < 4; r++) acc[i][j][c][r] = 0.0;

        for(int kt = w.kt0; kt < w.kt1; kt++) {
            const bool more = lu < p.units;
            const int  slot_n = slot_r + 1 == ST ? 0 : slot_r + 1;
#pragma unroll
            for(int ks = 0; ks < NK; ks++) {
                const int f = ks & 1;
                if(ks == NK - 1) {
                    // the next k-tile has landed for every thread, and every warp has read this tile's last fragments:
                    // its slot is the one the next round of copies overwrites
                    cp_async_commit();
                    cp_async_wait<ST - 2>();
                    __syncthreads();
                    load_frag(f ^ 1, slot_n, 0);
                } else {
                    load_frag(f ^ 1, slot_r, (ks + 1) * 4);
                    if(more) {
#pragma unroll
                        for(int q = ks * NCOPY / (NK - 1); q < (ks + 1) * NCOPY / (NK - 1); q++) load_copy(q, slot_w);
                    }
                }
                double sa[MT][2], sb[NT];  // ar + ai, br + bi of the 3M product
                if constexpr(CPLX) {
#pragma unroll
                    for(int i = 0; i < MT; i++) {
                        sa[i][0] = fa[f][i][0].x + fa[f][i][0].y;
                        sa[i][1] = fa[f][i][1].x + fa[f][i][1].y;
                    }
#pragma unroll
                    for(int j = 0; j < NT; j++) sb[j] = fb[f][j].x + fb[f][j].y;
                }
#pragma unroll
                for(int i = 0; i < MT; i++)
#pragma unroll
                    for(int j = 0; j < NT; j++) {
                        if constexpr(!CPLX) {
                            dmma(acc[i][j][0], fa[f][i][0], fa[f][i][1], fb[f][j]);
                        } else {
                            dmma(acc[i][j][0], fa[f][i][0].x, fa[f][i][1].x, fb[f][j].x);  // t1 += ar br
                            dmma(acc[i][j][1], fa[f][i][0].y, fa[f][i][1].y, fb[f][j].y);  // t2 += ai bi
                            dmma(acc[i][j][2], sa[i][0], sa[i][1], sb[j]);                 // t3 += (ar + ai)(br + bi)
                        }
                    }
            }
            if(more) load_next();
            slot_w = slot_w + 1 == ST ? 0 : slot_w + 1;
            slot_r = slot_n;
        }

        auto value = [&](int i, int j, int r) -> T {
            if constexpr(!CPLX) {
                return acc[i][j][0][r];
            } else {
                const double t1 = acc[i][j][0][r], t2 = acc[i][j][1][r], t3 = acc[i][j][2][r];
                return make_double2(t1 - t2, t3 - t1 - t2);
            }
        };
        if(w.piece >= 0) {
            // Tail piece: the raw partial tile, element e = (i NT + j) 4 + r of thread tid at e * THR + tid
            // (coalesced), summed by gemm_split_reduce_kernel.
            T *P = reinterpret_cast<T *>(p.part) + (size_t)w.piece * (BM * BN);
#pragma unroll
            for(int i = 0; i < MT; i++)
#pragma unroll
                for(int j = 0; j < NT; j++)
#pragma unroll
                    for(int r = 0; r < 4; r++) P[((i * NT + j) * 4 + r) * THR + tid] = value(i, j, r);
            continue;
        }
        int tile_m, tile_n;
        gemm_raster<BM, BN>(w.tile, M, N, tile_m, tile_n);
        const int  m0 = tile_m * BM + wm0 + g, n0 = tile_n * BN + wn0 + 2 * t;
        T         *C        = reinterpret_cast<T *>(p.C) + (int64_t)w.bz * p.sC;
        const bool use_beta = (p.beta.x != 0.0) || (p.beta.y != 0.0);
        // C = alpha * v + beta * C at tile element (i, j, r) (C is not read when beta == 0)
        auto put = [&](int i, int j, int r, T v) {
            const int gm = m0 + i * 16 + ((r >> 1) << 3), gn = n0 + j * 8 + (r & 1);
            if(gm < M && gn < N) {
                T *cp = C + gm + (int64_t)gn * p.ldc;
                if constexpr(!CPLX) {
                    double o = p.alpha.x * v;
                    if(use_beta) o += p.beta.x * (*cp);
                    *cp = o;
                } else {
                    double2 o = cmul(p.alpha, v);
                    if(use_beta) o = cadd(o, cmul(p.beta, *cp));
                    *cp = o;
                }
            }
        };
        if(p.cluster <= 1) {
#pragma unroll
            for(int i = 0; i < MT; i++)
#pragma unroll
                for(int j = 0; j < NT; j++)
#pragma unroll
                    for(int r = 0; r < 4; r++) put(i, j, r, value(i, j, r));
            continue;
        }
        // Cluster split: every CTA leaves its partial tile in its own shared memory, then sums one share of the tile
        // over the cluster in rank (= K) order through distributed shared memory.
        cp_async_wait<0>();
        __syncthreads();
#pragma unroll
        for(int i = 0; i < MT; i++)
#pragma unroll
            for(int j = 0; j < NT; j++)
#pragma unroll
                for(int r = 0; r < 4; r++) smem[((i * NT + j) * 4 + r) * THR + tid] = value(i, j, r);
        asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
        constexpr int EPT  = MT * NT * 4;
        const int     rank = u % p.cluster;
        for(int e = EPT * rank / p.cluster; e < EPT * (rank + 1) / p.cluster; e++) {
            const uint32_t own = smem0 + (uint32_t)((e * THR + tid) * sizeof(T));
            T              v{};
            for(int q = 0; q < p.cluster; q++) {
                uint32_t rem;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(rem) : "r"(own), "r"(q));
                if constexpr(!CPLX) {
                    double x;
                    asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(x) : "r"(rem) : "memory");
                    v = q == 0 ? x : v + x;
                } else {
                    double x, y;
                    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];\n" : "=d"(x), "=d"(y) : "r"(rem) : "memory");
                    v = q == 0 ? make_double2(x, y) : make_double2(v.x + x, v.y + y);
                }
            }
            put((e >> 2) / NT, (e >> 2) % NT, e & 3, v);
        }
        asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");  // no CTA leaves while its tile is read
        return;
    }
}

// Second pass of the tail split: sums each tail tile's `split` partial pieces in piece order (the same order on
// every run) and writes C = alpha * sum + beta * C with the GEMM kernel's thread mapping.  Grid: (tail tiles,
// EPT / EPB); each thread takes EPB of its tile elements and issues all EPB * split loads before any addition,
// so the pass runs at memory bandwidth instead of one load latency per partial.
constexpr int SPLIT_MAX   = 16;
constexpr int CLUSTER_MAX = 4;
template<bool CPLX, int CFG>
struct SplitReduce {
    using G                  = GemmTile<CPLX, CFG>;
    static constexpr int MT = G::WM / 16, NT = G::WN / 8;
    static constexpr int EPT = MT * NT * 4;   // tile elements per thread
    static constexpr int EPB = CPLX ? 2 : 4;  // elements per thread per CTA of the reduction
};
template<bool CPLX, int CFG>
__global__ void __launch_bounds__(GemmTile<CPLX, CFG>::THREADS) gemm_split_reduce_kernel(const GemmArgs p) {
    grid_wait();
    using G  = GemmTile<CPLX, CFG>;
    using T  = typename Scalar<CPLX>::T;
    using SR = SplitReduce<CPLX, CFG>;
    constexpr int BM = G::BM, BN = G::BN, WM = G::WM, WN = G::WN, NT = SR::NT, EPB = SR::EPB, THR = G::THREADS;
    const int     tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int     g = lane >> 2, t = lane & 3;
    const int     wm0 = (warp % (BM / WM)) * WM, wn0 = (warp / (BM / WM)) * WN;
    const int     tail = blockIdx.x, e0 = blockIdx.y * EPB;
    const int     tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN), bz = (p.nfull + tail) / tiles;
    int           tile_m, tile_n;
    gemm_raster<BM, BN>((p.nfull + tail) % tiles, p.M, p.N, tile_m, tile_n);
    const int     m0 = tile_m * BM, n0 = tile_n * BN;
    const T      *P  = reinterpret_cast<const T *>(p.part) + (size_t)tail * p.split * (BM * BN);
    T            *C  = reinterpret_cast<T *>(p.C) + (int64_t)bz * p.sC;
    const bool    use_beta = (p.beta.x != 0.0) || (p.beta.y != 0.0);
    const int     ns = p.split < SPLIT_MAX ? p.split : SPLIT_MAX;
    T             w[EPB][SPLIT_MAX];
#pragma unroll
    for(int q = 0; q < SPLIT_MAX; q++)
#pragma unroll
        for(int u = 0; u < EPB; u++)
            if(q < ns) w[u][q] = P[(size_t)q * (BM * BN) + (e0 + u) * THR + tid];
#pragma unroll
    for(int u = 0; u < EPB; u++) {
        const int e = e0 + u, r = e & 3, j = (e >> 2) % NT, i = (e >> 2) / NT;
        T         v = w[u][0];
#pragma unroll
        for(int q = 1; q < SPLIT_MAX; q++)
            if(q < ns) {
                if constexpr(!CPLX)
                    v += w[u][q];
                else
                    v = cadd(v, w[u][q]);
            }
        const int gm = m0 + wm0 + i * 16 + g + ((r >> 1) << 3);
        const int gn = n0 + wn0 + j * 8 + 2 * t + (r & 1);
        if(gm < p.M && gn < p.N) {
            T *cp = C + gm + (int64_t)gn * p.ldc;
            if constexpr(!CPLX) {
                double o = p.alpha.x * v;
                if(use_beta) o += p.beta.x * (*cp);
                *cp = o;
            } else {
                double2 o = cmul(p.alpha, v);
                if(use_beta) o = cadd(o, cmul(p.beta, *cp));
                *cp = o;
            }
        }
    }
}

// Bytes of tail-split scratch that let every GEMM of a matvec-sized problem pick its best split: at most
// 4 * (co-resident CTAs) partial tiles of the larger (real) tile.
size_t gemm_split_ws_bytes();

// Host launcher.  Returns HEFF_OK or a status code; never synchronises.
template<bool CPLX>
int gemm_f64(bool ta, bool tb, const GemmArgs &args, cudaStream_t stream);
bool gemm_fn_known(const void *f);  // a DMMA GEMM or split-reduction kernel (single GemmArgs parameter)

}  // namespace heff
