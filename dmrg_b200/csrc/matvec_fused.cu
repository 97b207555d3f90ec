// H_eff * theta in one launch, for bonds whose four-stage product is bound by its chain of launches and latencies.
#include <algorithm>
#include "matvec.cuh"
#include "runtime.cuh"

namespace heff {

// A cluster of `cl` CTAs owns eight consecutive a'; its CTA of rank r owns the columns b in [r bs, (r + 1) bs) of theta.
//   G1   T1[m,s][a' + 8 b]  = sum_a x[(s,b), a] L[a, (m,a')]   rows (s,b), one n-tile of eight a' per m
//   MIX  T2[n,b][s' + S a'] = sum_{m,s} T1 W                   points (a',b) x entries of W
//   G2   y[b', (s',a')]    += sum_{(n,b)} R[(n,b), b'] T2      this CTA's b only
// The eight a' need nothing of the others', and a CTA's b stay in its shared memory through the three products, so the only
// exchange is the sum of G2's partial results: 16-byte pushes to the CTA of the cluster that owns the column b', summed there
// in rank order.  All three products run on the FP64 tensor pipe (complex: four real products).  Operands are read once into
// shared memory, R's part behind G1 and the mix; R is read through strides, in the caller's layout or the permuted one.
// A zero weight of W must not touch its input (0 * inf): a CTA that finds a non-finite T1 mixes entry by entry.
struct FusedArgs {
    const void *x, *L, *R, *W;
    void       *y;
    int64_t     r_n, r_bp;                        // R[b + r_bp b' + r_n n]
    int         S, cL, cR, DL, DR, cl, bs;
    int         px, pl, pk, p1, p2;               // pitches: x per b, L per (m,a'), R per b', T1 per (m,s), T2 per (n,b)
    int         oL, oR, oF, o1, o2, bytes;        // shared memory: x, L (then the partial sums), R, fragments of W, T1, T2
    bool        vx, vl, vr;                       // 16-byte copies (real)
};
constexpr int FU_THR = 512, FU_SMEM = 227 * 1024;

template<bool CPLX>
static bool fused_plan(const MatvecDims &d, FusedArgs &a) {
    const int es = CPLX ? 16 : 8, per = CPLX ? 8 : 16;  // shared-memory banks in elements
    a.S = (int)d.S, a.cL = (int)d.cL, a.cR = (int)d.cR, a.DL = (int)d.DL, a.DR = (int)d.DR;
    a.cl = 8;
    while(a.cl > 1 && a.cR < 4 * a.cl) a.cl >>= 1;
    a.bs          = (int)((cdiv(a.cR, a.cl) + 1) / 2 * 2);
    auto pitch    = [&](int64_t n, int r) { while(n % per != r) n++; return (int)n; };
    auto up       = [](int64_t n, int64_t q) { return (n + q - 1) / q * q; };
    const int K1  = (int)up(a.cL, 4), K2 = (int)up((int64_t)a.DR * a.bs, 4), KM = (int)up((int64_t)a.DL * a.S, 4);
    a.px          = pitch((int64_t)a.S * K1, a.S == 1 ? 4 : (CPLX ? 0 : 8));
    a.pl          = pitch(K1, 4);
    a.pk          = pitch(K2, 4);
    auto plane    = [&](int64_t n) { while(n % 16 != 4) n++; return (int)n; };  // T1, T2: planes of doubles
    a.p1          = plane(8 * a.bs);
    a.p2          = plane(8 * a.S);
    const int64_t nx = (int64_t)a.bs * a.px, nl = (int64_t)a.DL * 8 * a.pl, nred = (int64_t)a.cl * cdiv(a.cR, a.cl) * 8 * a.S;
    const int64_t nr = up(a.cR, 16) * a.pk, nf = (int64_t)(KM / 4) * cdiv((int64_t)a.DR * a.S, 8) * 32;
    const int64_t n1 = (int64_t)KM * a.p1, n2 = (int64_t)K2 * a.p2;
    const int64_t oR = std::max(nx + nl, up(nred, 2)), oF = oR + nr, o1 = oF + nf, o2 = o1 + n1, tot = o2 + n2;
    if(tot * es > FU_SMEM) return false;
    a.oL = (int)nx * es, a.oR = (int)oR * es, a.oF = (int)oF * es, a.o1 = (int)o1 * es, a.o2 = (int)o2 * es, a.bytes = (int)tot * es;
    return true;
}

__device__ __forceinline__ bool fu_bad(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

// 16 x 8 tile over nk steps of four, d = A B with fragments fa(ks, half) and fb(ks); complex: its real (part 0) or imaginary part.
// Two accumulator sets halve the chain.
template<bool CX, class FA, class FB>
__device__ __forceinline__ void fu_tile(int nk, int part, FA fa, FB fb, double (&d)[4]) {
    double e[4] = {0, 0, 0, 0};
#pragma unroll
    for(int u = 0; u < 4; u++) d[u] = 0.0;
#pragma unroll 4
    for(int ks = 0; ks < nk; ks++) {
        const auto a0 = fa(ks, 0), a1 = fa(ks, 1), b = fb(ks);
        if constexpr(!CX) {
            if(ks & 1)
                dmma(e, a0, a1, b);
            else
                dmma(d, a0, a1, b);
        } else {
            dmma(d, a0.x, a1.x, part ? b.y : b.x);
            dmma(e, a0.y, a1.y, part ? b.x : -b.y);
        }
    }
#pragma unroll
    for(int u = 0; u < 4; u++) d[u] += e[u];
}

template<class T>
__global__ void __launch_bounds__(FU_THR) matvec_fused_kernel(const FusedArgs a) {
    grid_wait();
    constexpr bool CX = sizeof(T) == 16;
    extern __shared__ __align__(16) unsigned char fu_smem[];
    T           *sx = reinterpret_cast<T *>(fu_smem), *sl = reinterpret_cast<T *>(fu_smem + a.oL), *sr = reinterpret_cast<T *>(fu_smem + a.oR);
    T           *sf = reinterpret_cast<T *>(fu_smem + a.oF);
    double      *s1 = reinterpret_cast<double *>(fu_smem + a.o1), *s2 = reinterpret_cast<double *>(fu_smem + a.o2);
    const int    thr = blockDim.x, warps = thr >> 5, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int    S = a.S, cL = a.cL, cR = a.cR, bs = a.bs;
    const int    rank = (int)blockIdx.x % a.cl, a0 = (int)blockIdx.x / a.cl * 8, na = min(8, cL - a0);
    const int    b0 = rank * bs, nb = max(0, min(bs, cR - b0));
    const T     *x = reinterpret_cast<const T *>(a.x), *L = reinterpret_cast<const T *>(a.L), *R = reinterpret_cast<const T *>(a.R);
    const T     *W = reinterpret_cast<const T *>(a.W);
    T            z;
    if constexpr(CX)
        z = make_double2(0.0, 0.0);
    else
        z = 0.0;
    // rows of `len` elements (zeros up to `pad`) from src + row * stride; one warp copies 32 chunks of a row at a time
    auto rows = [&](T *dst, int pitch, const T *src, int64_t stride, int nrow, int nvalid, int len, int pad, bool vec) {
        const int E = !CX && vec ? 2 : 1, nch = (pad + 32 * E - 1) / (32 * E);
        for(int i = warp; i < nrow * nch; i += warps) {
            const int r = i / nch, e = (i - r * nch) * 32 * E + lane * E;
            if(e >= pad) continue;
            const bool ok = r < nvalid && e < len;
            const T   *p  = ok ? src + stride * r + e : src;
            if(CX || E == 2)
                cp_async<16>(smem_u32(dst + r * pitch + e), p, ok);
            else
                cp_async<(int)sizeof(T)>(smem_u32(dst + r * pitch + e), p, ok);
        }
    };
    const int K1 = (cL + 3) / 4 * 4, K2 = (a.DR * bs + 3) / 4 * 4, KS = (a.DL * S + 3) / 4, NT = (a.DR * S + 7) / 8;
    rows(sx, a.px, nb > 0 ? x + (int64_t)S * cL * b0 : x, (int64_t)S * cL, bs, nb, S * cL, S * K1, a.vx);
    for(int m = 0; m < a.DL; m++) rows(sl + m * 8 * a.pl, a.pl, L + (int64_t)cL * (a0 + (int64_t)cL * m), cL, 8, na, cL, K1, a.vl);
    cp_async_commit();
    {
        const int E = !CX && a.vr ? 2 : 1, cR16 = (cR + 15) / 16 * 16;
        for(int e = lane * E; e < K2; e += 32 * E) {
            const int  n = e / bs, bl = e - n * bs;
            const bool ok = n < a.DR && bl < nb;
            const T   *p  = ok ? R + a.r_n * n + b0 + bl : R;
            for(int r = warp; r < cR16; r += warps) {
                const bool v = ok && r < cR;
                const T   *q = v ? p + a.r_bp * r : R;
                if(CX || E == 2)
                    cp_async<16>(smem_u32(sr + r * a.pk + e), q, v);
                else
                    cp_async<(int)sizeof(T)>(smem_u32(sr + r * a.pk + e), q, v);
            }
        }
    }
    cp_async_commit();
    bool wim = false;
    for(int e = tid; e < KS * NT * 32; e += thr) {  // W as DMMA fragments: entry (i = m S + s, o = n S + s')
        const int f = e >> 5, i = (f / NT) * 4 + (e & 3), o = (f % NT) * 8 + ((e & 31) >> 2);
        T         v = z;
        if(i < a.DL * S && o < a.DR * S) {
            const int m = i / S, s = i - m * S, n = o / S, so = o - n * S;
            v = W[m + a.DL * (n + a.DR * (s + S * so))];
        }
        sf[e] = v;
        if constexpr(CX) wim = wim || v.y != 0.0;
    }
    constexpr int NP  = CX ? 2 : 1;  // planes (and tasks) of a complex tile
    const int     pl1 = 4 * KS * a.p1, pl2 = K2 * a.p2;
    for(int p = 0; p < NP; p++) {
        for(int e = tid; e < (4 * KS - a.DL * S) * a.p1; e += thr) s1[p * pl1 + a.DL * S * a.p1 + e] = 0.0;
        for(int e = tid; e < (K2 - a.DR * bs) * a.p2; e += thr) s2[p * pl2 + a.DR * bs * a.p2 + e] = 0.0;
    }
    cp_async_wait<1>();
    if constexpr(CX)
        wim = __syncthreads_or(wim) != 0;
    else
        __syncthreads();

    bool bad = false;
    {  // G1
        const int R1 = S * bs, MT = (R1 + 15) / 16;
        for(int task = warp; task < MT * a.DL * NP; task += warps) {
            const int part = CX ? task & 1 : 0, tt = task / NP, mt = tt / a.DL, m = tt - mt * a.DL;
            const int r0 = 16 * mt + g, r1 = r0 + 8, c0 = min(r0, R1 - 1), c1 = min(r1, R1 - 1);
            const T  *x0 = sx + (c0 / S) * a.px + c0 % S + t * S, *x1 = sx + (c1 / S) * a.px + c1 % S + t * S;
            const T  *lb = sl + (m * 8 + g) * a.pl + t;
            double    d[4];
            fu_tile<CX>(
                K1 / 4, part, [&](int ks, int h) { return (h ? x1 : x0)[4 * ks * S]; }, [&](int ks) { return lb[4 * ks]; }, d);
#pragma unroll
            for(int h = 0; h < 2; h++) {
                const int r = h ? r1 : r0;
                if(r >= R1) continue;
                const int    bl = r / S, s = r - bl * S;
                const double v0 = bl < nb ? d[2 * h] : 0.0, v1 = bl < nb ? d[2 * h + 1] : 0.0;
                bad             = bad || fu_bad(v0) || fu_bad(v1);
                *reinterpret_cast<double2 *>(s1 + part * pl1 + (m * S + s) * a.p1 + 8 * bl + 2 * t) = make_double2(v0, v1);
            }
        }
    }
    bad = __syncthreads_or(bad) != 0;
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");  // x and L have been read: partial sums may land there
    if(!bad) {  // MIX
        const int PT = bs / 2;
        for(int task = warp; task < PT * NT * NP; task += warps) {
            const int     part = CX ? task & 1 : 0, tt = task / NP, pt = tt / NT, nt = tt - pt * NT;
            const double *pa = s1 + t * a.p1 + 16 * pt + g;
            const T      *pb = sf + nt * 32 + lane;
            double        d[4];
            if constexpr(CX) {
                if(wim)
                    fu_tile<true>(
                        KS, part, [&](int ks, int h) { return make_double2(pa[4 * ks * a.p1 + 8 * h], pa[pl1 + 4 * ks * a.p1 + 8 * h]); },
                        [&](int ks) { return pb[ks * NT * 32]; }, d);
                else
                    fu_tile<false>(
                        KS, 0, [&](int ks, int h) { return pa[part * pl1 + 4 * ks * a.p1 + 8 * h]; }, [&](int ks) { return pb[ks * NT * 32].x; }, d);
            } else {
                fu_tile<false>(
                    KS, 0, [&](int ks, int h) { return pa[4 * ks * a.p1 + 8 * h]; }, [&](int ks) { return pb[ks * NT * 32]; }, d);
            }
#pragma unroll
            for(int c = 0; c < 2; c++) {
                const int o = 8 * nt + 2 * t + c;
                if(o >= a.DR * S) continue;
                const int n = o / S, so = o - n * S;
#pragma unroll
                for(int h = 0; h < 2; h++)  // rows g, g + 8: a' = g of b = 2 pt + h
                    s2[part * pl2 + (n * bs + 2 * pt + h) * a.p2 + so + S * g] = d[2 * h + c];
            }
        }
    } else {
        for(int e = tid; e < a.DR * S * 8 * bs; e += thr) {
            const int p = e % (8 * bs), o = e / (8 * bs), n = o / S, so = o - n * S;
            double    re = 0.0, im = 0.0;
            for(int i = 0; i < a.DL * S; i++) {
                const int    m = i / S, s = i - m * S;
                const T      w = W[m + a.DL * (n + a.DR * (s + S * so))];
                const double v = s1[i * a.p1 + p];
                if constexpr(CX) {
                    const double u = s1[pl1 + i * a.p1 + p];
                    if(w.x != 0.0 || w.y != 0.0) re = fma(w.x, v, fma(-w.y, u, re)), im = fma(w.x, u, fma(w.y, v, im));
                } else {
                    if(w != 0.0) re = fma(w, v, re);
                }
            }
            const int i2 = (n * bs + p / 8) * a.p2 + so + S * (p % 8);
            s2[i2]       = re;
            if constexpr(CX) s2[pl2 + i2] = im;
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    const int CO = (cR + a.cl - 1) / a.cl, R2 = 8 * S, plr = a.cl * CO * R2;  // columns b' per owner, rows of a column
    double   *red = reinterpret_cast<double *>(sx);                           // (part, source rank, column, row)
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");     // every CTA is past G1
    {  // G2
        const int MT = (cR + 15) / 16;
        for(int task = warp; task < MT * S * NP; task += warps) {
            const int     part = CX ? task & 1 : 0, tt = task / NP, mt = tt / S, q = tt - mt * S;
            const T      *pa = sr + (16 * mt + g) * a.pk + t;
            const double *pb = s2 + t * a.p2 + 8 * q + g;
            double        d[4];
            fu_tile<CX>(
                K2 / 4, part, [&](int ks, int h) { return pa[4 * ks + 8 * h * a.pk]; },
                [&](int ks) {
                    if constexpr(CX)
                        return make_double2(pb[4 * ks * a.p2], pb[pl2 + 4 * ks * a.p2]);
                    else
                        return pb[4 * ks * a.p2];
                },
                d);
#pragma unroll
            for(int h = 0; h < 2; h++) {
                const int bp = 16 * mt + g + 8 * h;
                if(bp >= cR) continue;
                uint32_t addr;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                             : "=r"(addr)
                             : "r"(smem_u32(red + part * plr + (rank * CO + bp / a.cl) * R2 + 8 * q + 2 * t)), "r"(bp % a.cl));
                asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};\n" ::"r"(addr), "d"(d[2 * h]), "d"(d[2 * h + 1]) : "memory");
            }
        }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    T *y = reinterpret_cast<T *>(a.y);
    for(int e = tid; e < CO * R2; e += thr) {
        const int r2 = e % R2, c = e / R2, bp = c * a.cl + rank;
        if(bp >= cR || r2 >= S * na) continue;
        double re = red[e], im = CX ? red[plr + e] : 0.0;
        for(int q = 1; q < a.cl; q++) {
            re += red[q * CO * R2 + e];
            if constexpr(CX) im += red[plr + q * CO * R2 + e];
        }
        T *dst = y + (int64_t)S * (a0 + (int64_t)cL * bp) + r2;
        if constexpr(CX)
            *dst = make_double2(re, im);
        else
            *dst = re;
    }
}

// Taken where one wave of clusters does the whole product and no CTA has much to do: the four kernels then wait for launches and
// latencies (us, four kernels / fused, D = 3: real S = 4 chi = 16 10.6 / 5.8, 48 12.9 / 7.7, 96 15.0 / 11.0; complex S = 4
// 48 18.4 / 10.8, 96 21.8 / 21.9; complex S = 2 96 x 128 19.8 / 16.4; D = 9 real S = 4 32 22.8 / 9.9, 64 24.6 / 14.7).  Clusters of
// eight CTAs that fill an SM each start on about two thirds of the SMs at a time (real S = 4 chi = 128 would take two waves:
// 17.9 / 25.5).  A CTA alone in its cluster also stages all of its x and L alone: complex S = 4 252 x 5, 592k multiply-adds,
// 17.0 / 17.8, hence the smaller bound there.
template<bool CPLX>
bool matvec_fused_fits(const MatvecDims &d) {
    FusedArgs a{};
    if(d.cL > 4096 || d.cR > 4096 || !fused_plan<CPLX>(d, a)) return false;
    const int64_t wave = (int64_t)device_sm_count() * 2 / 3, ctas = cdiv(d.cL, 8) * a.cl, per_sm = a.bytes <= 113 * 1024 ? 2 : 1;
    const int64_t work = (CPLX ? 4 : 1) * 8 * d.S * (a.bs * d.DL * d.cL + d.cR * d.DR * a.bs);  // real multiply-adds of a CTA
    return ctas <= wave * per_sm && work * (ctas > wave ? 2 : 1) <= 500000 + 25000 * a.cl;
}

template<bool CPLX>
int matvec_fused(const MatvecDims &d, const typename Scalar<CPLX>::T *x, typename Scalar<CPLX>::T *y, const typename Scalar<CPLX>::T *L,
                 const typename Scalar<CPLX>::T *R, int64_t r_n, int64_t r_bp, const typename Scalar<CPLX>::T *W, cudaStream_t s) {
    using T = typename Scalar<CPLX>::T;
    FusedArgs a{};
    if(!fused_plan<CPLX>(d, a)) return HEFF_BAD_SHAPE;
    a.x = x, a.L = L, a.R = R, a.W = W, a.y = y, a.r_n = r_n, a.r_bp = r_bp;
    auto al = [](const void *p) { return ((uintptr_t)p & 15u) == 0; };
    a.vx    = !CPLX && al(x) && (d.S * d.cL) % 2 == 0;
    a.vl    = !CPLX && al(L) && d.cL % 2 == 0;
    a.vr    = !CPLX && al(R) && r_n % 2 == 0 && r_bp % 2 == 0 && d.cR % 2 == 0;
    static int attr_done[64] = {0};
    int        dev           = 0;
    HEFF_CUDA(cudaGetDevice(&dev));
    if(dev < 0 || dev >= 64 || !attr_done[dev]) {
        HEFF_CUDA(cudaFuncSetAttribute(matvec_fused_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, FU_SMEM));
        if(dev >= 0 && dev < 64) attr_done[dev] = 1;
    }
    // 16 warps where a product has more than eight tiles per CTA, else eight (0.3 us less in barriers)
    const int64_t np = CPLX ? 2 : 1, t1 = np * cdiv(d.S * a.bs, 16) * d.DL, tm = np * (a.bs / 2) * cdiv(d.DR * d.S, 8), t2 = np * cdiv(d.cR, 16) * d.S;
    const int     thr = std::max(t1, std::max(tm, t2)) > 8 ? FU_THR : FU_THR / 2;
    HEFF_CUDA((launch_chained_cluster((unsigned)a.cl, matvec_fused_kernel<T>, dim3((unsigned)(cdiv(d.cL, 8) * a.cl)), dim3((unsigned)thr), (size_t)a.bytes, s, a)));
    count_launches(1);
    return HEFF_OK;
}
template bool matvec_fused_fits<false>(const MatvecDims &);
template bool matvec_fused_fits<true>(const MatvecDims &);
template int  matvec_fused<false>(const MatvecDims &, const double *, double *, const double *, const double *, int64_t, int64_t, const double *, cudaStream_t);
template int  matvec_fused<true>(const MatvecDims &, const double2 *, double2 *, const double2 *, const double2 *, int64_t, int64_t, const double2 *,
                                cudaStream_t);

}  // namespace heff
