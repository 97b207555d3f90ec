// Host-side dispatch of the DMMA GEMM template (gemm_f64.cuh).
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "gemm_f64.cuh"
#include "runtime.cuh"

namespace heff {

// Tail-split mode of the DMMA GEMMs: 0 no K split at all, 1 automatic (the cost model below), 2..16 that many pieces
// whenever the large tiles leave a partial wave.  Initial value from the environment variable HEFF_GEMM_SPLIT (default 1).
static std::atomic<int> g_split_mode{-1};

static int split_mode() {
    int m = g_split_mode.load();
    if(m < 0) {
        const char *e      = getenv("HEFF_GEMM_SPLIT");
        const int   v      = e ? atoi(e) : 1;
        int         expect = -1;
        g_split_mode.compare_exchange_strong(expect, (v >= 0 && v <= 16) ? v : 1);
        m = g_split_mode.load();
    }
    return m;
}

size_t gemm_split_ws_bytes() {
    // at most 4 partial tiles per co-resident CTA (the real kernel runs one 128x128 CTA per SM)
    return (size_t)4 * device_sm_count() * GemmTile<false, 0>::BM * GemmTile<false, 0>::BN * sizeof(double);
}

// Every DMMA GEMM kernel (and split reduction) this process has launched; a captured graph's kernel nodes are
// recognised by their function (their one parameter is a GemmArgs), so a replay can retarget their output.
static std::mutex               g_gemm_fn_mu;
static std::vector<const void *> g_gemm_fns;
static void gemm_fn_register(const void *f) {
    std::lock_guard<std::mutex> lk(g_gemm_fn_mu);
    if(std::find(g_gemm_fns.begin(), g_gemm_fns.end(), f) == g_gemm_fns.end()) g_gemm_fns.push_back(f);
}
bool gemm_fn_known(const void *f) {
    std::lock_guard<std::mutex> lk(g_gemm_fn_mu);
    return std::find(g_gemm_fns.begin(), g_gemm_fns.end(), f) != g_gemm_fns.end();
}

// How a GEMM runs: tile shape; K pieces of every tile on a cluster (cluster > 1); or K pieces of the tiles of the last
// partial wave, from tile nfull on, summed by a second kernel (split > 1).  Tiles count over all batch members.
struct GemmPlan {
    int     cfg = 0, cluster = 1, split = 1;
    int64_t nfull = 0;
    double  cost  = 0;
};

struct TileShape {
    int    bm, bn, bk, occ;  // co-resident CTAs per SM
    double full, alone;      // sustained fraction of the DMMA rate: SM full of such CTAs, one CTA alone on its SM
};
template<bool CPLX>
static const TileShape &tile_shape(int cfg) {
    static const TileShape r[3] = {{128, 128, 32, 1, 0.95, 0.95}, {64, 64, 32, 1, 0.92, 0.92}, {32, 32, 32, 3, 0.86, 0.62}};
    static const TileShape c[2] = {{64, 64, 32, 1, 0.87, 0.87}, {32, 32, 32, 2, 0.82, 0.65}};
    return CPLX ? c[cfg] : r[cfg];
}

// Plan of one problem: the smallest estimate over tile shapes and K splits.  An SM does 64 DMMA FMAs per clock
// whatever the tile, so a variant's time is the busiest SM's share of the padded products at the rate its tile sustains
// (tile_shape), plus what its launches cost.  The constants come from a sweep of every variant over the matvec and
// environment GEMMs of chi = 8 .. 1024 (real / complex): a cluster of 2 or 4 adds 3.6 us (8 adds 7 and never won), the chained
// reduction kernel of a tail split 3 us (at 5, its price as a plain launch, whole tiles were kept too long: real S = 4
// 313 x 569 178 / 154 us, S = 2 307 x 525 92 / 88).  Examples, us for (whole tiles
// of 128/64/32 | best): f64 96x128x32 10.3/6.2/4.2 | 4.2; f64 1024x256x768 109/31/18.5 | 18.5; c128 192x128x384
// -/49/18.5 | 10.3 (cluster of 4); f64 3072x4096x1024 840/-/- | 743 (tail split).
template<bool CPLX>
static GemmPlan gemm_pick(const GemmArgs &a) {
    constexpr double kClk = 1.9e9, kLaunch = 3.2e-6, kCluster = 3.6e-6, kReduce = 3e-6, kHbm = 6.0e12;
    const int     mode = split_mode(), sms = device_sm_count();
    const double  fma  = CPLX ? 3.0 : 1.0;
    GemmPlan      best;
    bool          have = false;
    for(int cfg = 0; cfg < gemm_cfgs(CPLX); cfg++) {
        if(mode >= 2 && cfg > 0) break;  // forced tail split: the large tiles
        const TileShape &t     = tile_shape<CPLX>(cfg);
        const int64_t    tiles = cdiv(a.M, t.bm) * cdiv(a.N, t.bn) * a.batch, KT = cdiv(a.K, t.bk);
        const double     kt_s  = (double)t.bm * t.bn * t.bk * fma / 64.0 / kClk;  // one k-tile at the full DMMA rate
        auto             rate  = [&](int64_t units) {
            const int64_t per = std::min<int64_t>(cdiv(units, sms), t.occ);
            return t.occ > 1 ? t.alone + (t.full - t.alone) * (double)(per - 1) / (t.occ - 1) : t.full;
        };
        for(int ks = 1; ks <= CLUSTER_MAX; ks *= 2) {
            const int64_t units = tiles * ks;
            // clusters are placed within a GPC: with one CTA per SM, a quarter of the SMs can stay out of reach of them
            if(ks > 1 && (mode != 1 || ks > KT || units > (t.occ > 1 ? sms : 3 * sms / 4))) break;
            GemmPlan q;
            q.cfg = cfg, q.cluster = ks, q.nfull = tiles;
            q.cost = kLaunch + (double)(cdiv(units, sms) * cdiv(KT, ks)) * kt_s / rate(units) + (ks > 1 ? kCluster : 0.0);
            if(!have || q.cost < best.cost) best = q, have = true;
        }
        if(t.occ == 1 && a.split_ws && mode >= 1 && tiles % sms != 0) {
            const double  unit_bytes = (double)t.bm * t.bn * (CPLX ? 16.0 : 8.0);
            const int64_t rem = tiles % sms, max_units = (int64_t)((double)a.split_ws_bytes / unit_bytes);
            for(int sp = mode >= 2 ? mode : 2; sp <= (mode >= 2 ? mode : SPLIT_MAX); sp++) {
                if(rem * sp > max_units || KT < (mode >= 2 ? sp : 4 * sp)) break;
                GemmPlan q;
                q.cfg = cfg, q.split = sp, q.nfull = tiles - rem;
                q.cost = kLaunch + (double)(tiles / sms * KT + cdiv(rem * sp, sms) * cdiv(KT, sp)) * kt_s / rate(tiles - rem + rem * sp) + kReduce +
                         2.0 * unit_bytes * (double)(rem * sp) / kHbm;
                if(q.cost < best.cost || mode >= 2) best = q;
            }
        }
    }
    return best;
}

template<bool CPLX, int CFG, bool TA, bool TB, int VEC>
static int launch_gemm(const GemmArgs &a_in, const GemmPlan &pl, cudaStream_t stream) {
    using G                  = GemmTile<CPLX, CFG>;
    using SM                 = GemmSmem<CPLX, CFG, TA, TB>;
    auto       kern = gemm_f64_kernel<CPLX, CFG, TA, TB, VEC>;
    static int occ[64] = {0};  // per instantiation and device: co-resident CTAs per SM (0 = not set up yet)
    int        dev     = 0;
    HEFF_CUDA(cudaGetDevice(&dev));
    if(dev < 0 || dev >= 64 || !occ[dev]) {
        HEFF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM::BYTES));
        int n = 0;
        HEFF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, G::THREADS, SM::BYTES));
        if(dev >= 0 && dev < 64) occ[dev] = n > 0 ? n : 1;
    }
    const int     per_sm = (dev >= 0 && dev < 64) ? occ[dev] : 1;
    const int64_t tiles  = cdiv(a_in.M, G::BM) * cdiv(a_in.N, G::BN) * a_in.batch;
    GemmArgs      a      = a_in;
    const int64_t units  = pl.cluster > 1 ? tiles * pl.cluster : pl.nfull + (tiles - pl.nfull) * pl.split;
    if(tiles > 0x3fffffffLL || units > 0x3fffffffLL) return HEFF_BAD_SHAPE;
    a.split   = pl.split;
    a.nfull   = (int)pl.nfull;
    a.part    = pl.split > 1 ? a.split_ws : nullptr;
    a.cluster = pl.cluster;
    a.units   = (int)units;
    gemm_fn_register(reinterpret_cast<const void *>(kern));
    // a cluster launch has one CTA per unit; otherwise one persistent CTA per slot at most
    const int64_t slots = pl.cluster > 1 ? units : (int64_t)device_sm_count() * per_sm;
    HEFF_CUDA(launch_chained_cluster((unsigned)pl.cluster, kern, (unsigned)std::min(units, slots), G::THREADS, SM::BYTES, stream, a));
    count_launches(pl.split > 1 ? 2 : 1);
    if(pl.split > 1) {
        using SR = SplitReduce<CPLX, CFG>;
        const dim3 rgrid((unsigned)(tiles - pl.nfull), (unsigned)(SR::EPT / SR::EPB));
        gemm_fn_register(reinterpret_cast<const void *>(gemm_split_reduce_kernel<CPLX, CFG>));
        HEFF_CUDA((launch_chained(gemm_split_reduce_kernel<CPLX, CFG>, rgrid, G::THREADS, 0, stream, a)));
    }
    return HEFF_OK;
}

template<bool CPLX, int CFG, int VEC>
static int launch_ops(bool ta, bool tb, const GemmArgs &a, const GemmPlan &pl, cudaStream_t s) {
    if(ta && tb) return HEFF_BAD_ARG;  // no caller forms A^T B^T
    if(ta) return launch_gemm<CPLX, CFG, true, false, VEC>(a, pl, s);
    if(tb) return launch_gemm<CPLX, CFG, false, true, VEC>(a, pl, s);
    return launch_gemm<CPLX, CFG, false, false, VEC>(a, pl, s);
}

static bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

template<bool CPLX, int VEC>
static int launch_plan(bool ta, bool tb, const GemmArgs &a, const GemmPlan &pl, cudaStream_t s) {
    if(pl.cfg == 0) return launch_ops<CPLX, 0, VEC>(ta, tb, a, pl, s);
    if(pl.cfg == 1) return launch_ops<CPLX, 1, VEC>(ta, tb, a, pl, s);
    if constexpr(!CPLX) return launch_ops<CPLX, 2, VEC>(ta, tb, a, pl, s);
    return HEFF_BAD_ARG;
}

template<>
int gemm_f64<false>(bool ta, bool tb, const GemmArgs &a, cudaStream_t s) {
    if(a.M <= 0 || a.N <= 0 || a.batch <= 0) return HEFF_OK;
    if(a.K <= 0) return HEFF_BAD_ARG;  // callers never form empty contractions
    // 16-byte copies need: 16B-aligned bases, even leading dims / batch strides, even contiguous extent.
    const bool v2 = aligned16(a.A) && aligned16(a.B) && (a.lda % 2 == 0) && (a.ldb % 2 == 0) && (a.sA % 2 == 0) && (a.sB % 2 == 0) &&
                    ((ta ? a.K : a.M) % 2 == 0) && ((tb ? a.N : a.K) % 2 == 0);
    const GemmPlan pl = gemm_pick<false>(a);
    return v2 ? launch_plan<false, 2>(ta, tb, a, pl, s) : launch_plan<false, 1>(ta, tb, a, pl, s);
}

template<>
int gemm_f64<true>(bool ta, bool tb, const GemmArgs &a, cudaStream_t s) {
    if(a.M <= 0 || a.N <= 0 || a.batch <= 0) return HEFF_OK;
    if(a.K <= 0) return HEFF_BAD_ARG;
    if(!aligned16(a.A) || !aligned16(a.B)) return HEFF_BAD_ARG;  // complex128 buffers are always 16-byte aligned
    return launch_plan<true, 1>(ta, tb, a, gemm_pick<true>(a), s);
}

}  // namespace heff

extern "C" int heff_gemm_set_tail_split(int mode) {
    if(mode < 0 || mode > heff::SPLIT_MAX) return -1;
    const int prev = heff::split_mode();
    heff::g_split_mode.store(mode);
    return prev;
}
