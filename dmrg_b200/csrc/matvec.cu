// H_eff * theta: layout kernels, MPO mixing kernel, matvec driver, expectation value,
// and the stateless C entry points heff_matvec_{d,z} / heff_expval_{d,z}.
#include <algorithm>
#include <initializer_list>
#include "matvec.cuh"
#include "runtime.cuh"
#include "wlist.cuh"

namespace heff {

int check_matvec_dims(const int64_t md[3], const int64_t wd[4], const int64_t ld[3], const int64_t rd[3], MatvecDims &d) {
    if(!md || !wd || !ld || !rd) return HEFF_BAD_ARG;
    d = MatvecDims{md[0], md[1], md[2], wd[0], wd[1]};
    // contraction_tblis.cpp:230-234
    if(md[1] != ld[0] || md[2] != rd[0] || md[0] != wd[2] || ld[2] != wd[0] || rd[2] != wd[1]) {
        set_last_error_msg("matvec: dimension mismatch mps [%lld,%lld,%lld] mpo [%lld,%lld,%lld,%lld] envL [%lld,%lld,%lld] envR [%lld,%lld,%lld]",
                           (long long)md[0], (long long)md[1], (long long)md[2], (long long)wd[0], (long long)wd[1], (long long)wd[2],
                           (long long)wd[3], (long long)ld[0], (long long)ld[1], (long long)ld[2], (long long)rd[0], (long long)rd[1],
                           (long long)rd[2]);
        return HEFF_BAD_SHAPE;
    }
    if(wd[3] != wd[2] || ld[1] != ld[0] || rd[1] != rd[0]) {
        set_last_error_msg("matvec: mpo must be [mL,mR,d,d] and envs [chi,chi,m]");
        return HEFF_BAD_SHAPE;
    }
    if(d.S <= 0 || d.cL <= 0 || d.cR <= 0 || d.DL <= 0 || d.DR <= 0) return HEFF_BAD_SHAPE;
    if(d.S > 64 || d.DL * d.S > 256 || d.DR * d.S > 256) {
        set_last_error_msg("matvec: spin*mpo bond dimension above 256 is not supported");
        return HEFF_BAD_SHAPE;
    }
    if(d.cL > (1 << 20) || d.cR > (1 << 20)) return HEFF_BAD_SHAPE;
    return HEFF_OK;
}

// x'[a + cL*(s + S*b)] = x[s + S*(a + cL*b)].  For the spins of one and two sites a thread moves the S values of a point (a, b),
// 16 bytes a load where x allows it, into S streams of consecutive a: one division per point, and whole sectors on both sides.
// Other spins go output-linear, one value and two divisions per thread.  us, output-linear / by points: real S = 4
// 1000 x 1000 20.0 / 10.9, 367 x 251 5.7 / 4.0, complex S = 4 1024 x 1024 25.5 / 17.8.
template<class T, int S>
__device__ __forceinline__ void permute_points(const T *__restrict__ x, T *__restrict__ xp, int64_t cL, int64_t points) {
    const bool vec = sizeof(T) == 8 && ((uintptr_t)x & 15u) == 0;
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < points; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = points <= 0x7fffffff ? (int64_t)((unsigned)e / (unsigned)cL) : e / cL, a = e - cL * b;
        T             v[S];
        if(vec) {
#pragma unroll
            for(int s = 0; s < S; s += 2) {
                const double2 w = *reinterpret_cast<const double2 *>(x + S * e + s);
                *reinterpret_cast<double *>(&v[s]) = w.x, *reinterpret_cast<double *>(&v[s + 1]) = w.y;
            }
        } else {
#pragma unroll
            for(int s = 0; s < S; s++) v[s] = x[S * e + s];
        }
#pragma unroll
        for(int s = 0; s < S; s++) xp[a + cL * (s + S * b)] = v[s];
    }
}
template<class T>
__global__ void permute_mps_kernel(const T *__restrict__ x, T *__restrict__ xp, int64_t S, int64_t cL, int64_t n) {
    grid_wait();
    if(S == 4) return permute_points<T, 4>(x, xp, cL, n / 4);
    if(S == 2) return permute_points<T, 2>(x, xp, cL, n / 2);
    for(int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < n; o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = o % cL, r = o / cL, s = r % S, b = r / S;
        xp[o]           = x[s + S * (a + cL * b)];
    }
}

// x'[o] for o in [o0, o1) (the x' columns (s,b) of a slab of b)
template<class T>
__global__ void permute_mps_range_kernel(const T *__restrict__ x, T *__restrict__ xp, int64_t S, int64_t cL, int64_t o0, int64_t o1) {
    grid_wait();
    for(int64_t o = o0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < o1; o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = o % cL, r = o / cL, s = r % S, b = r / S;
        xp[o]           = x[s + S * (a + cL * b)];
    }
}

// R'[b + cR*n + cR*DR*b'] = R[b + cR*(b' + cR*n)]
template<class T>
__global__ void permute_R_kernel(const T *__restrict__ R, T *__restrict__ Rp, int64_t cR, int64_t DR, int64_t n) {
    grid_wait();
    for(int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < n; o += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = o % cR, r = o / cR, nn = r % DR, bp = r / DR;
        Rp[o]           = R[b + cR * (bp + cR * nn)];
    }
}

__device__ __forceinline__ bool is_zero(double w) { return w == 0.0; }
__device__ __forceinline__ bool is_zero(double2 w) { return w.x == 0.0 && w.y == 0.0; }
__device__ __forceinline__ double fma_s(double w, double v, double acc) { return fma(w, v, acc); }
__device__ __forceinline__ double2 fma_s(double2 w, double2 v, double2 acc) {
    return make_double2(fma(w.x, v.x, fma(-w.y, v.y, acc.x)), fma(w.x, v.y, fma(w.y, v.x, acc.y)));
}
__device__ __forceinline__ void zero(double &v) { v = 0.0; }
__device__ __forceinline__ void zero(double2 &v) { v = make_double2(0.0, 0.0); }

// MPO mix (MixArgs, matvec.cuh) on the FP64 tensor pipe: at 16 points of a warp, out (16 x J S) = in (16 x K S) W.  The
// dense product costs less than walking W's nonzero entries (~20 % in spin chains) with a shared-memory load or two per
// multiply-add: 6 DMMAs per 16 points for the two-site Ising MPO (D = 3), 45 for its square, and the kernel stays bound by
// HBM for large tensors and by its two dependent memory latencies for small ones.  W is laid out once per CTA as DMMA
// fragments; a CTA owns TP consecutive points p and walks q in steps of gridDim.y with the next tile in flight.  Two
// accumulator columns are two consecutive s', so eight points' stores of one (j, s') pair fill whole sectors.
// A zero weight must not touch its input: the reference skips zero entries, and 0 * inf would not.  A warp that meets a
// non-finite input computes its points entry by entry instead (mix_skip).
// us before / after: chi = 16 real D = 3 10.6 / 5.2, chi = 1024 complex D = 3 114 / 89 (HBM floor 62), real D = 9 367 x 251
// 53 / 26, environment real D = 9 640 x 517 165 / 43 Larger MPOs too, whole product, real 256 x 256, from the nonzero list / dense:
// S = 16 D = 3 (72 fragments of W) 247 / 156, S = 4 D = 16 (128) 387 / 191, S = 8 D = 9 (162) 430 / 221; complex S = 16 D = 3
// 559 / 448.
template<class T>
__device__ __noinline__ void mix_skip(const MixArgs &a, const T *tile, int pitch, int p, int q, int o0, int o1) {
    const int S = a.S, NI = a.K * S;
    const T  *W = reinterpret_cast<const T *>(a.W);
    for(int o = o0; o < o1; o++) {
        const int j = o / S, so = o - j * S;
        T         acc;
        zero(acc);
        for(int i = 0; i < NI; i++) {
            const int k = a.s_fastest ? i / S : i % a.K, s = a.s_fastest ? i % S : i / a.K;
            const T   w = W[(int64_t)a.w_k * k + (int64_t)a.w_j * j + (int64_t)a.w_s * s + (int64_t)a.w_so * so];
            if(!is_zero(w)) acc = fma_s(w, tile[(k * S + s) * pitch], acc);
        }
        reinterpret_cast<T *>(a.out)[so + (int64_t)S * (p + (int64_t)a.P * (q + (int64_t)a.Q * j))] = acc;
    }
}

__device__ __forceinline__ bool non_finite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ bool non_finite(double2 v) { return non_finite(v.x) || non_finite(v.y); }

template<class T, int TP>
struct MixTile {
    static constexpr bool CX    = sizeof(T) == 16;
    static constexpr int  THR   = 2 * TP;                // one warp per 16 points
    static constexpr int  PITCH = TP + (CX ? 2 : 4);     // conflict-free fragment loads
};
template<class T, int TP, int NTC>
__global__ void __launch_bounds__(2 * TP) mix_dense_kernel(const MixArgs a) {
    grid_wait();
    using MT = MixTile<T, TP>;
    constexpr bool CX = MT::CX;
    constexpr int  THR = MT::THR, WARPS = THR / 32, PITCH = MT::PITCH;
    extern __shared__ __align__(16) unsigned char mix_smem[];
    const int    S = a.S, NI = a.K * S, NO = a.J * S, KS = (NI + 3) / 4, NT = (NO + 7) / 8;
    T           *tile = reinterpret_cast<T *>(mix_smem);                 // a.bufs tiles of 4 KS x PITCH (rows past NI are zero)
    T           *frag = tile + (size_t)a.bufs * 4 * KS * PITCH;          // (ks, nt, lane)
    const T     *in   = reinterpret_cast<const T *>(a.in), *W = reinterpret_cast<const T *>(a.W);
    T           *out  = reinterpret_cast<T *>(a.out);
    const int    tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int    p0 = blockIdx.x * TP, np = min(TP, a.P - p0);
    auto load = [&](int q, int buf) {
        T       *dst = tile + (size_t)buf * 4 * KS * PITCH;
        const T *src = in + p0 + a.in_q * q;
        for(int i = warp; i < 4 * KS; i += WARPS) {
            const int  k = i / S, s = i - k * S;
            const bool row = i < NI;
            const T   *r   = src + a.in_k * k + a.in_s * s;
            if(CX || a.vec) {
                constexpr int E = CX ? 1 : 2;
                for(int p = lane * E; p < TP; p += 32 * E) cp_async<16>(smem_u32(dst + i * PITCH + p), row && p < np ? r + p : in, row && p < np);
            } else {
                for(int p = lane; p < TP; p += 32) cp_async<(int)sizeof(T)>(smem_u32(dst + i * PITCH + p), row && p < np ? r + p : in, row && p < np);
            }
        }
        cp_async_commit();
    };
    int q = a.q0 + (int)blockIdx.y;
    load(q, 0);
    bool wim = false;  // W has an imaginary part
    for(int e = tid; e < KS * NT * 32; e += THR) {
        const int f = e >> 5, i = (f / NT) * 4 + (e & 3), o = (f % NT) * 8 + ((e & 31) >> 2);
        T         v;
        zero(v);
        if(i < NI && o < NO) {
            const int k = i / S, s = i - k * S, j = o / S, so = o - j * S;
            v = W[(int64_t)a.w_k * k + (int64_t)a.w_j * j + (int64_t)a.w_s * s + (int64_t)a.w_so * so];
        }
        frag[e] = v;
        if constexpr(CX) wim = wim || v.y != 0.0;
    }
    if constexpr(CX) wim = __syncthreads_or(wim) != 0;
    const int     pw = warp * 16;                       // this warp's points of the tile
    const int64_t jstep = (int64_t)S * a.P * a.Q;
    for(int buf = 0; q < a.q0 + a.nq; q += (int)gridDim.y, buf ^= a.bufs - 1) {
        const int qn = q + (int)gridDim.y;
        if(a.bufs == 2) {
            if(qn < a.q0 + a.nq)
                load(qn, buf ^ 1);
            else
                cp_async_commit();
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const T *x   = tile + (size_t)buf * 4 * KS * PITCH + pw;
        bool     bad = false;
        if(pw < np) {
            for(int n0 = 0; n0 < NT; n0 += NTC) {
                double re[NTC][4], im[CX ? NTC : 1][4];
#pragma unroll
                for(int n = 0; n < NTC; n++)
#pragma unroll
                    for(int u = 0; u < 4; u++) {
                        re[n][u] = 0.0;
                        if constexpr(CX) im[n][u] = 0.0;
                    }
#pragma unroll 2
                for(int ks = 0; ks < KS; ks++) {
                    const T a0 = x[(4 * ks + t) * PITCH + g], a1 = x[(4 * ks + t) * PITCH + g + 8];
                    bad        = bad || non_finite(a0) || non_finite(a1);
                    const T *fr = frag + (size_t)(ks * NT + n0) * 32 + lane;
#pragma unroll
                    for(int n = 0; n < NTC; n++)
                        if(n0 + n < NT) {
                            const T b = fr[n * 32];
                            if constexpr(!CX) {
                                dmma(re[n], a0, a1, b);
                            } else {
                                dmma(re[n], a0.x, a1.x, b.x);
                                dmma(im[n], a0.y, a1.y, b.x);
                                if(wim) {
                                    dmma(re[n], -a0.y, -a1.y, b.y);
                                    dmma(im[n], a0.x, a1.x, b.y);
                                }
                            }
                        }
                }
                if(__any_sync(0xffffffffu, bad)) break;
#pragma unroll
                for(int n = 0; n < NTC; n++) {
                    const int o = (n0 + n) * 8 + 2 * t;
                    if(o >= NO) continue;
                    const int j = o / S, so = o - j * S;
#pragma unroll
                    for(int h = 0; h < 2; h++) {
                        const int p = pw + g + 8 * h;
                        if(p >= np) continue;
                        T *dst = out + so + jstep * j + (int64_t)S * (p0 + p + (int64_t)a.P * q);
                        T  v0, v1;
                        if constexpr(!CX)
                            v0 = re[n][2 * h], v1 = re[n][2 * h + 1];
                        else
                            v0 = make_double2(re[n][2 * h], im[n][2 * h]), v1 = make_double2(re[n][2 * h + 1], im[n][2 * h + 1]);
                        if(!CX && a.pairs) {
                            if constexpr(!CX) *reinterpret_cast<double2 *>(dst) = make_double2(v0, v1);
                        } else {
                            dst[0] = v0;
                            if(o + 1 < NO) (so + 1 < S ? dst + 1 : dst - so + jstep)[0] = v1;
                        }
                    }
                }
            }
            if(__any_sync(0xffffffffu, bad)) {  // lanes 0..15 and 16..31 take half of the outputs each, a point per lane
                const int p = pw + (lane & 15), half = (NO + 1) / 2;
                if(p < np) mix_skip<T>(a, x + (lane & 15), PITCH, p0 + p, q, lane < 16 ? 0 : half, lane < 16 ? half : NO);
            }
        }
        __syncthreads();  // the tile has been read
        if(a.bufs == 1 && qn < a.q0 + a.nq) load(qn, 0);
    }
}

// Entry by entry: environment MPOs whose input rows do not fit a tile of 32 points (K S of about 700 real, 300 complex and more).
// One thread per point, bound by the chain of its loads; W in shared memory, in the order of the sum, so an entry costs a load and
// a test (read from global memory and its indices by division: environment d = 2 1024 -> 1 at chi = 64 936 us, now 457).
constexpr size_t MIX_SMEM = 200 * 1024;
template<class T>
__global__ void __launch_bounds__(128) mix_entry_kernel(const MixArgs a) {
    grid_wait();
    extern __shared__ __align__(16) unsigned char mix_smem[];
    T            *sW = reinterpret_cast<T *>(mix_smem);  // (output, input)
    const T      *W  = reinterpret_cast<const T *>(a.W);
    const int     S = a.S, NI = a.K * S, NO = a.J * S;
    const int     n1 = a.s_fastest ? a.K : S, n2 = a.s_fastest ? S : a.K;  // outer and inner index of the sum
    const int64_t d1 = a.s_fastest ? a.in_k : a.in_s, d2 = a.s_fastest ? a.in_s : a.in_k;
    for(int e = threadIdx.x; e < NI * NO; e += blockDim.x) {
        const int o = e / NI, i = e - o * NI, j = o / S, so = o - j * S, i1 = i / n2, i2 = i - i1 * n2;
        const int k = a.s_fastest ? i1 : i2, s = a.s_fastest ? i2 : i1;
        sW[e] = W[(int64_t)a.w_k * k + (int64_t)a.w_j * j + (int64_t)a.w_s * s + (int64_t)a.w_so * so];
    }
    __syncthreads();
    for(int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)a.P * a.nq; e += (int64_t)gridDim.x * blockDim.x) {
        const int p = (int)(e % a.P), q = a.q0 + (int)(e / a.P);
        const T  *x = reinterpret_cast<const T *>(a.in) + p + a.in_q * q, *w = sW;
        T        *out = reinterpret_cast<T *>(a.out) + (int64_t)S * (p + (int64_t)a.P * q);
        for(int j = 0; j < a.J; j++)
            for(int so = 0; so < S; so++) {
                T acc;
                zero(acc);
                for(int i1 = 0; i1 < n1; i1++) {
                    const T *xi = x + d1 * i1;
                    for(int i2 = 0; i2 < n2; i2++, w++)
                        if(!is_zero(*w)) acc = fma_s(*w, xi[d2 * i2], acc);
                }
                out[so + (int64_t)S * a.P * a.Q * j] = acc;
            }
    }
}

template<class T, int TP>
static size_t mix_bytes(const MixArgs &a, int bufs) {
    const size_t KS = (size_t)cdiv((int64_t)a.K * a.S, 4), NT = (size_t)cdiv((int64_t)a.J * a.S, 8);
    return sizeof(T) * (bufs * 4 * KS * MixTile<T, TP>::PITCH + KS * NT * 32);
}
template<class T, int TP, int NTC>
static int mix_launch(const MixArgs &a, cudaStream_t s) {
    const size_t smem = mix_bytes<T, TP>(a, a.bufs);
    static int   attr_done[64] = {0};
    int          dev           = 0;
    HEFF_CUDA(cudaGetDevice(&dev));
    if(dev < 0 || dev >= 64 || !attr_done[dev]) {
        HEFF_CUDA(cudaFuncSetAttribute(mix_dense_kernel<T, TP, NTC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MIX_SMEM));
        if(dev >= 0 && dev < 64) attr_done[dev] = 1;
    }
    // about as many CTAs as the device holds; each then lays W out once for several q
    const int64_t tx  = cdiv(a.P, TP);
    const int64_t occ = std::max<int64_t>(1, std::min<int64_t>(1024 / MixTile<T, TP>::THR, (int64_t)(224 * 1024 / (smem + 1024))));
    const int64_t ny  = std::min<int64_t>(a.nq, std::max<int64_t>(1, (int64_t)device_sm_count() * occ / tx));
    HEFF_CUDA((launch_chained(mix_dense_kernel<T, TP, NTC>, dim3((unsigned)tx, (unsigned)ny), MixTile<T, TP>::THR, smem, s, a)));
    return HEFF_OK;
}
// Two tiles in flight where two such CTAs fit an SM.
template<class T, int TP>
static int mix_tiles(MixArgs a, cudaStream_t s) {
    a.bufs = mix_bytes<T, TP>(a, 2) <= 110 * 1024 ? 2 : 1;
    return cdiv((int64_t)a.J * a.S, 8) <= 2 ? mix_launch<T, TP, 2>(a, s) : mix_launch<T, TP, 5>(a, s);
}
// Points per tile: 128, fewer while that leaves SMs without a CTA or the tile does not fit.
template<bool CPLX>
int mpo_mix(MixArgs a, cudaStream_t s) {
    using T = typename Scalar<CPLX>::T;
    if(a.nq <= 0 || a.P <= 0) return HEFF_OK;
    a.pairs = !CPLX && a.S % 2 == 0 && ((uintptr_t)a.out & 15u) == 0;
    a.vec   = !CPLX && ((uintptr_t)a.in & 15u) == 0 && a.P % 2 == 0 && a.in_k % 2 == 0 && a.in_s % 2 == 0 && a.in_q % 2 == 0;
    if(mix_bytes<T, 32>(a, 1) > MIX_SMEM) {
        const size_t  wsm = sizeof(T) * (size_t)a.K * a.J * a.S * a.S;
        const int64_t n = (int64_t)a.P * a.nq, g = std::min<int64_t>(cdiv(n, 128), (int64_t)device_sm_count() * 16);
        if(wsm > MIX_SMEM) return HEFF_BAD_SHAPE;  // neither operators nor environments accept such an MPO
        if(wsm > 48 * 1024) HEFF_CUDA(cudaFuncSetAttribute(mix_entry_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MIX_SMEM));
        HEFF_CUDA((launch_chained(mix_entry_kernel<T>, (unsigned)g, 128, wsm, s, a)));
        return HEFF_OK;
    }
    auto padded = [&](int tp) { return cdiv(a.P, tp) * tp; };
    int  TP     = 128;
    if(cdiv(a.P, 128) * a.nq < 2 * device_sm_count() || mix_bytes<T, 128>(a, 1) > MIX_SMEM || 16 * padded(128) > 17 * padded(64)) TP = 64;
    if(TP == 64 && (cdiv(a.P, 64) * a.nq < 2 * device_sm_count() || mix_bytes<T, 64>(a, 1) > MIX_SMEM || 16 * padded(64) > 17 * padded(32))) TP = 32;
    if(TP == 128) return mix_tiles<T, 128>(a, s);
    if(TP == 64) return mix_tiles<T, 64>(a, s);
    return mix_tiles<T, 32>(a, s);
}
template int mpo_mix<false>(MixArgs, cudaStream_t);
template int mpo_mix<true>(MixArgs, cudaStream_t);

static int grid_1d(int64_t n) {
    int64_t g = (n + 255) / 256;
    int64_t cap = (int64_t)device_sm_count() * 16;
    return (int)(g < cap ? (g > 0 ? g : 1) : cap);
}

template<bool CPLX>
int permute_R(const typename Scalar<CPLX>::T *R, typename Scalar<CPLX>::T *Rp, const MatvecDims &d, cudaStream_t s) {
    const int64_t n = d.size_Rp();
    HEFF_CUDA((launch_chained(permute_R_kernel<typename Scalar<CPLX>::T>, grid_1d(n), 256, 0, s, R, Rp, d.cR, d.DR, n)));
    return HEFF_OK;
}

// limit on the MPO's size: W, its nonzero list and 128 points of T1 within 200 KB
template<bool CPLX>
static bool mpo_too_large(const MatvecDims &d) {
    const size_t es = CPLX ? 16 : 8;
    return es * ((size_t)d.DL * d.DR * d.S * d.S + (size_t)d.DL * d.S * 128) + wlist_bytes((int)d.DL, (int)d.DR, (int)d.S, es) > 200 * 1024;
}

// T2[(s' + S a') + S cL (b + cR n)] = sum_{m,s} W[m + DL(n + DR(s + S s'))] T1[(a' + cL m) + cL DL (s + S b)], b0 <= b < b0 + nb
template<bool CPLX>
static int launch_mix(const MatvecDims &d, const typename Scalar<CPLX>::T *T1, typename Scalar<CPLX>::T *T2, const typename Scalar<CPLX>::T *W,
                      cudaStream_t s, int64_t b0 = 0, int64_t nb = -1) {
    using T = typename Scalar<CPLX>::T;
    if(mpo_too_large<CPLX>(d)) return HEFF_BAD_SHAPE;
    if(nb < 0) nb = d.cR;
    if(nb > 65535) return HEFF_BAD_SHAPE;
    MixArgs a{};
    a.in = T1, a.out = T2, a.W = W;
    a.K = (int)d.DL, a.J = (int)d.DR, a.S = (int)d.S, a.P = (int)d.cL, a.Q = (int)d.cR, a.q0 = (int)b0, a.nq = (int)nb;
    a.in_k = d.cL, a.in_s = d.cL * d.DL, a.in_q = d.cL * d.DL * d.S;
    a.w_k = 1, a.w_j = (int)d.DL, a.w_s = (int)(d.DL * d.DR), a.w_so = (int)(d.DL * d.DR * d.S);
    return mpo_mix<CPLX>(a, s);
}

template<bool CPLX>
int matvec_fp64(const MatvecDims &d, const typename Scalar<CPLX>::T *x, typename Scalar<CPLX>::T *y, const typename Scalar<CPLX>::T *L,
                const typename Scalar<CPLX>::T *Rp, const typename Scalar<CPLX>::T *W, const MatvecScratch<CPLX> &ws, cudaStream_t s,
                cudaEvent_t *ev) {
    const int64_t n = d.size_mps();
    if(!ev && matvec_fused_fits<CPLX>(d)) {
        if(mpo_too_large<CPLX>(d)) return HEFF_BAD_SHAPE;
        return matvec_fused<CPLX>(d, x, y, L, Rp, d.cR, d.cR * d.DR, W, s);
    }
    if(ev) HEFF_CUDA(cudaEventRecord(ev[0], s));
    HEFF_CUDA((launch_chained(permute_mps_kernel<typename Scalar<CPLX>::T>, grid_1d(n), 256, 0, s, x, ws.xp, d.S, d.cL, n)));
    count_launches(2);  // the permutation and the MPO mix below (the GEMM launcher counts its own kernels)
    if(ev) HEFF_CUDA(cudaEventRecord(ev[1], s));
    GemmArgs g1{};
    g1.M     = (int)(d.cL * d.DL);
    g1.N     = (int)(d.S * d.cR);
    g1.K     = (int)d.cL;
    g1.batch = 1;
    g1.A     = L;
    g1.lda   = d.cL;
    g1.B     = ws.xp;
    g1.ldb   = d.cL;
    g1.C     = ws.T1;
    g1.ldc   = d.cL * d.DL;
    g1.alpha = make_double2(1.0, 0.0);
    g1.beta  = make_double2(0.0, 0.0);
    g1.split_ws       = ws.split_ws;
    g1.split_ws_bytes = ws.split_bytes;
    HEFF_TRY(gemm_f64<CPLX>(/*ta=*/true, /*tb=*/false, g1, s));
    if(ev) HEFF_CUDA(cudaEventRecord(ev[2], s));
    HEFF_TRY(launch_mix<CPLX>(d, ws.T1, ws.T2, W, s));
    if(ev) HEFF_CUDA(cudaEventRecord(ev[3], s));
    GemmArgs g2{};
    g2.M     = (int)(d.S * d.cL);
    g2.N     = (int)d.cR;
    g2.K     = (int)(d.cR * d.DR);
    g2.batch = 1;
    g2.A     = ws.T2;
    g2.lda   = d.S * d.cL;
    g2.B     = Rp;
    g2.ldb   = d.cR * d.DR;
    g2.C     = y;
    g2.ldc   = d.S * d.cL;
    g2.alpha = make_double2(1.0, 0.0);
    g2.beta  = make_double2(0.0, 0.0);
    g2.split_ws       = ws.split_ws;
    g2.split_ws_bytes = ws.split_bytes;
    HEFF_TRY(gemm_f64<CPLX>(false, false, g2, s));
    if(ev) HEFF_CUDA(cudaEventRecord(ev[4], s));
    return HEFF_OK;
}

// First two stages of the matvec with alpha folded into GEMM 1 and the mix written to `out`:
//   out[s' + S (a' + cL (b + cR n))] = alpha * sum_{a,m,s} L[a,a',m] x[s,a,b] W[m,n,s,s']
// which is the L-side subspace-expansion term P of EnvBase::get_expansion_term (EnvBase.cpp:303-333).
template<bool CPLX>
int matvec_left_stages(const MatvecDims &d, const typename Scalar<CPLX>::T *x, const typename Scalar<CPLX>::T *L, const typename Scalar<CPLX>::T *W,
                       typename Scalar<CPLX>::T *out, typename Scalar<CPLX>::T *xp, typename Scalar<CPLX>::T *T1, double alpha, cudaStream_t s) {
    const int64_t n = d.size_mps();
    HEFF_CUDA((launch_chained(permute_mps_kernel<typename Scalar<CPLX>::T>, grid_1d(n), 256, 0, s, x, xp, d.S, d.cL, n)));
    GemmArgs g1{};
    g1.M     = (int)(d.cL * d.DL);
    g1.N     = (int)(d.S * d.cR);
    g1.K     = (int)d.cL;
    g1.batch = 1;
    g1.A     = L;
    g1.lda   = d.cL;
    g1.B     = xp;
    g1.ldb   = d.cL;
    g1.C     = T1;
    g1.ldc   = d.cL * d.DL;
    g1.alpha = make_double2(alpha, 0.0);
    g1.beta  = make_double2(0.0, 0.0);
    HEFF_TRY(gemm_f64<CPLX>(/*ta=*/true, /*tb=*/false, g1, s));
    return launch_mix<CPLX>(d, T1, out, W, s);
}

// y = H_eff x with x and y in HOST memory, copies overlapped with the computation.  The slab of theta with
// columns b in [b0, b1) is contiguous (theta[s + S(a + cL b)]), and GEMM 1 and the mix of that slab need
// nothing else: slab c is copied in on the copy stream and processed on compute stream c % 2 as soon as it
// has landed.  GEMM 2's output columns b' are independent: slab c' of y is computed on stream c' % 2 once
// every mix is done and copied out right after.  Two compute streams let a slab's GEMM fill the tail wave of
// the previous one.  Synchronises before returning.
template<bool CPLX>
int matvec_fp64_host(const MatvecDims &d, const typename Scalar<CPLX>::T *xh, typename Scalar<CPLX>::T *yh, const typename Scalar<CPLX>::T *L,
                     const typename Scalar<CPLX>::T *Rp, const typename Scalar<CPLX>::T *W, const MatvecScratch<CPLX> &ws, typename Scalar<CPLX>::T *dx,
                     typename Scalar<CPLX>::T *dy, const HostPipe &hp) {
    using T               = typename Scalar<CPLX>::T;
    const int         nin = (int)std::min<int64_t>(hp.n_in, d.cR), nout = (int)std::min<int64_t>(hp.n_out, d.cR);
    cudaStream_t      cs[2] = {hp.s, hp.aux};
    const int64_t     colx = d.S * d.cL;  // elements per b column of theta / y
    auto              slab = [&](int c, int nc, int64_t &b0, int64_t &b1) {
        b0 = d.cR * c / nc;
        b1 = d.cR * (c + 1) / nc;
    };
    // everything queued on the caller's stream before this call precedes the copies into dx
    HEFF_CUDA(cudaEventRecord(hp.ev[0], hp.s));
    HEFF_CUDA(cudaStreamWaitEvent(hp.copy, hp.ev[0], 0));
    HEFF_CUDA(cudaStreamWaitEvent(hp.aux, hp.ev[0], 0));
    for(int c = 0; c < nin; c++) {
        int64_t b0, b1;
        slab(c, nin, b0, b1);
        if(b1 == b0) continue;
        HEFF_CUDA(cudaMemcpyAsync(dx + colx * b0, xh + colx * b0, sizeof(T) * colx * (b1 - b0), cudaMemcpyHostToDevice, hp.copy));
        HEFF_CUDA(cudaEventRecord(hp.ev[1 + c], hp.copy));
        cudaStream_t s = cs[c & 1];
        HEFF_CUDA(cudaStreamWaitEvent(s, hp.ev[1 + c], 0));
        const int64_t o0 = d.cL * d.S * b0, o1 = d.cL * d.S * b1;
        HEFF_CUDA((launch_chained(permute_mps_range_kernel<T>, grid_1d(o1 - o0), 256, 0, s, dx, ws.xp, d.S, d.cL, o0, o1)));
        GemmArgs g1{};
        g1.M = (int)(d.cL * d.DL), g1.N = (int)(d.S * (b1 - b0)), g1.K = (int)d.cL, g1.batch = 1;
        g1.A = L, g1.lda = d.cL, g1.B = ws.xp + o0, g1.ldb = d.cL, g1.C = ws.T1 + d.cL * d.DL * d.S * b0, g1.ldc = d.cL * d.DL;
        g1.alpha = make_double2(1.0, 0.0), g1.beta = make_double2(0.0, 0.0);
        HEFF_TRY(gemm_f64<CPLX>(/*ta=*/true, /*tb=*/false, g1, s));
        HEFF_TRY(launch_mix<CPLX>(d, ws.T1, ws.T2, W, s, b0, b1 - b0));
    }
    // every mix (both streams) before any GEMM 2 slab
    HEFF_CUDA(cudaEventRecord(hp.ev[HostPipe::MAXS + 1], hp.aux));
    HEFF_CUDA(cudaStreamWaitEvent(hp.s, hp.ev[HostPipe::MAXS + 1], 0));
    HEFF_CUDA(cudaEventRecord(hp.ev[HostPipe::MAXS + 2], hp.s));
    HEFF_CUDA(cudaStreamWaitEvent(hp.aux, hp.ev[HostPipe::MAXS + 2], 0));
    for(int c = 0; c < nout; c++) {
        int64_t b0, b1;
        slab(c, nout, b0, b1);
        if(b1 == b0) continue;
        cudaStream_t s = cs[c & 1];
        GemmArgs     g2{};
        g2.M = (int)(d.S * d.cL), g2.N = (int)(b1 - b0), g2.K = (int)(d.cR * d.DR), g2.batch = 1;
        g2.A = ws.T2, g2.lda = d.S * d.cL, g2.B = Rp + d.cR * d.DR * b0, g2.ldb = d.cR * d.DR, g2.C = dy + colx * b0, g2.ldc = d.S * d.cL;
        g2.alpha = make_double2(1.0, 0.0), g2.beta = make_double2(0.0, 0.0);
        HEFF_TRY(gemm_f64<CPLX>(false, false, g2, s));
        HEFF_CUDA(cudaEventRecord(hp.ev[HostPipe::MAXS + 3 + c], s));
        HEFF_CUDA(cudaStreamWaitEvent(hp.copy, hp.ev[HostPipe::MAXS + 3 + c], 0));
        HEFF_CUDA(cudaMemcpyAsync(yh + colx * b0, dy + colx * b0, sizeof(T) * colx * (b1 - b0), cudaMemcpyDeviceToHost, hp.copy));
    }
    // the caller's stream resumes after the last copy out; the host waits for it
    HEFF_CUDA(cudaEventRecord(hp.ev[2 * HostPipe::MAXS + 3], hp.copy));
    HEFF_CUDA(cudaStreamWaitEvent(hp.s, hp.ev[2 * HostPipe::MAXS + 3], 0));
    HEFF_CUDA(cudaStreamSynchronize(hp.s));
    return HEFF_OK;
}

// ---- deterministic dot product ----
constexpr int DOT_BLOCKS = 1024;
template<bool CPLX>
__global__ void dot_partial_kernel(const typename Scalar<CPLX>::T *__restrict__ x, const typename Scalar<CPLX>::T *__restrict__ y, int64_t n,
                                   double *partials) {
    grid_wait();
    __shared__ double sre[256], sim[256];
    double            re = 0, im = 0;
    for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if constexpr(CPLX) {
            double2 a = x[i], b = y[i];
            re += a.x * b.x + a.y * b.y;  // conj(a) * b
            im += a.x * b.y - a.y * b.x;
        } else {
            re += x[i] * y[i];
        }
    }
    sre[threadIdx.x] = re;
    sim[threadIdx.x] = im;
    __syncthreads();
    for(int w = 128; w > 0; w >>= 1) {
        if(threadIdx.x < w) {
            sre[threadIdx.x] += sre[threadIdx.x + w];
            sim[threadIdx.x] += sim[threadIdx.x + w];
        }
        __syncthreads();
    }
    if(threadIdx.x == 0) {
        partials[blockIdx.x]              = sre[0];
        partials[DOT_BLOCKS + blockIdx.x] = sim[0];
    }
}
template<bool CPLX>
__global__ void dot_final_kernel(const double *partials, int nb, typename Scalar<CPLX>::T *out) {
    grid_wait();
    __shared__ double sre[256], sim[256];
    double            re = 0, im = 0;
    for(int i = threadIdx.x; i < nb; i += 256) {
        re += partials[i];
        im += partials[DOT_BLOCKS + i];
    }
    sre[threadIdx.x] = re;
    sim[threadIdx.x] = im;
    __syncthreads();
    for(int w = 128; w > 0; w >>= 1) {
        if(threadIdx.x < w) {
            sre[threadIdx.x] += sre[threadIdx.x + w];
            sim[threadIdx.x] += sim[threadIdx.x + w];
        }
        __syncthreads();
    }
    if(threadIdx.x == 0) {
        if constexpr(CPLX)
            *out = make_double2(sre[0], sim[0]);
        else
            *out = sre[0];
    }
}

template<bool CPLX>
int dot_device(const typename Scalar<CPLX>::T *x, const typename Scalar<CPLX>::T *y, int64_t n, typename Scalar<CPLX>::T *out, double *partials,
               cudaStream_t s) {
    int nb = (int)std::min<int64_t>(DOT_BLOCKS, std::max<int64_t>(1, (n + 255) / 256));
    HEFF_CUDA((launch_chained(dot_partial_kernel<CPLX>, nb, 256, 0, s, x, y, n, partials)));
    HEFF_CUDA((launch_chained(dot_final_kernel<CPLX>, 1, 256, 0, s, partials, nb, out)));
    return HEFF_OK;
}

const void *permute_kernel_fn(bool cplx) {
    return cplx ? reinterpret_cast<const void *>(permute_mps_kernel<double2>) : reinterpret_cast<const void *>(permute_mps_kernel<double>);
}

template<bool CPLX>
int permute_mps(const MatvecDims &d, const typename Scalar<CPLX>::T *x, typename Scalar<CPLX>::T *xp, cudaStream_t s) {
    const int64_t n = d.size_mps();
    HEFF_CUDA((launch_chained(permute_mps_kernel<typename Scalar<CPLX>::T>, grid_1d(n), 256, 0, s, x, xp, d.S, d.cL, n)));
    return HEFF_OK;
}
template<bool CPLX>
int mix_fp64(const MatvecDims &d, const typename Scalar<CPLX>::T *T1, typename Scalar<CPLX>::T *T2, const typename Scalar<CPLX>::T *W, cudaStream_t s) {
    return launch_mix<CPLX>(d, T1, T2, W, s);
}
template int permute_mps<false>(const MatvecDims &, const double *, double *, cudaStream_t);
template int permute_mps<true>(const MatvecDims &, const double2 *, double2 *, cudaStream_t);
template int mix_fp64<false>(const MatvecDims &, const double *, double *, const double *, cudaStream_t);
template int mix_fp64<true>(const MatvecDims &, const double2 *, double2 *, const double2 *, cudaStream_t);
template int permute_R<false>(const double *, double *, const MatvecDims &, cudaStream_t);
template int permute_R<true>(const double2 *, double2 *, const MatvecDims &, cudaStream_t);
template int matvec_fp64<false>(const MatvecDims &, const double *, double *, const double *, const double *, const double *,
                                const MatvecScratch<false> &, cudaStream_t, cudaEvent_t *);
template int matvec_fp64<true>(const MatvecDims &, const double2 *, double2 *, const double2 *, const double2 *, const double2 *,
                               const MatvecScratch<true> &, cudaStream_t, cudaEvent_t *);
template int matvec_left_stages<false>(const MatvecDims &, const double *, const double *, const double *, double *, double *, double *, double,
                                       cudaStream_t);
template int matvec_left_stages<true>(const MatvecDims &, const double2 *, const double2 *, const double2 *, double2 *, double2 *, double2 *, double,
                                      cudaStream_t);
template int matvec_fp64_host<false>(const MatvecDims &, const double *, double *, const double *, const double *, const double *,
                                     const MatvecScratch<false> &, double *, double *, const HostPipe &);
template int matvec_fp64_host<true>(const MatvecDims &, const double2 *, double2 *, const double2 *, const double2 *, const double2 *,
                                    const MatvecScratch<true> &, double2 *, double2 *, const HostPipe &);
template int dot_device<false>(const double *, const double *, int64_t, double *, double *, cudaStream_t);
template int dot_device<true>(const double2 *, const double2 *, int64_t, double2 *, double *, cudaStream_t);

// ---- stateless entry points ----
// Complex tensors are read by 16-byte loads on every route (the GEMM refuses others, the one-launch product has no such test).
template<bool CPLX>
static int check_alignment(std::initializer_list<const void *> tensors) {
    for(const void *p : tensors)
        if(CPLX && ((uintptr_t)p & 15u)) {
            set_last_error_msg("matvec: complex tensors must be 16-byte aligned");
            return HEFF_BAD_ARG;
        }
    return HEFF_OK;
}

template<bool CPLX>
static int matvec_stateless(void *res, const void *mps, const int64_t md[3], const void *mpo, const int64_t wd[4], const void *envL,
                            const int64_t ld[3], const void *envR, const int64_t rd[3], cudaStream_t s) {
    using T = typename Scalar<CPLX>::T;
    MatvecDims d;
    HEFF_TRY(check_matvec_dims(md, wd, ld, rd, d));
    if(!res || !mps || !mpo || !envL || !envR) return HEFF_BAD_ARG;
    if(res == mps) {
        set_last_error_msg("matvec: res must not alias mps");
        return HEFF_BAD_ARG;
    }
    HEFF_TRY(check_alignment<CPLX>({res, mps, mpo, envL, envR}));
    if(matvec_fused_fits<CPLX>(d)) {  // R in the caller's layout
        if(mpo_too_large<CPLX>(d)) return HEFF_BAD_SHAPE;
        return matvec_fused<CPLX>(d, reinterpret_cast<const T *>(mps), reinterpret_cast<T *>(res), reinterpret_cast<const T *>(envL),
                                  reinterpret_cast<const T *>(envR), d.cR * d.cR, d.cR, reinterpret_cast<const T *>(mpo), s);
    }
    const int64_t elems = MatvecScratch<CPLX>::elems(d) + MatvecScratch<CPLX>::pad(d.size_Rp());
    const size_t  split = matvec_split_bytes((size_t)elems * sizeof(T));
    void         *base  = nullptr;
    HEFF_TRY(stream_workspace(s, (size_t)elems * sizeof(T) + split, &base));
    MatvecScratch<CPLX> ws;
    T                  *Rp = ws.carve(reinterpret_cast<T *>(base), d);
    ws.split_ws           = reinterpret_cast<unsigned char *>(base) + (size_t)elems * sizeof(T);
    ws.split_bytes        = split;
    HEFF_TRY(permute_R<CPLX>(reinterpret_cast<const T *>(envR), Rp, d, s));
    return matvec_fp64<CPLX>(d, reinterpret_cast<const T *>(mps), reinterpret_cast<T *>(res), reinterpret_cast<const T *>(envL), Rp,
                             reinterpret_cast<const T *>(mpo), ws, s);
}

template<bool CPLX>
static int expval_stateless(double *result, const void *mps, const int64_t md[3], const void *mpo, const int64_t wd[4], const void *envL,
                            const int64_t ld[3], const void *envR, const int64_t rd[3], cudaStream_t s) {
    using T = typename Scalar<CPLX>::T;
    MatvecDims d;
    HEFF_TRY(check_matvec_dims(md, wd, ld, rd, d));
    if(!result || !mps || !mpo || !envL || !envR) return HEFF_BAD_ARG;
    HEFF_TRY(check_alignment<CPLX>({mps, mpo, envL, envR}));
    const int64_t extra = MatvecScratch<CPLX>::pad(d.size_Rp()) + MatvecScratch<CPLX>::pad(d.size_mps()) + 1;
    const int64_t elems = MatvecScratch<CPLX>::elems(d) + extra;
    void         *base  = nullptr;
    HEFF_TRY(stream_workspace(s, (size_t)elems * sizeof(T) + 2 * DOT_BLOCKS * sizeof(double), &base));
    MatvecScratch<CPLX> ws;
    T      *Rp       = ws.carve(reinterpret_cast<T *>(base), d);
    T      *y        = Rp + MatvecScratch<CPLX>::pad(d.size_Rp());
    T      *dres     = y + d.size_mps();
    double *partials = reinterpret_cast<double *>(dres + 1);
    HEFF_TRY(permute_R<CPLX>(reinterpret_cast<const T *>(envR), Rp, d, s));
    HEFF_TRY(matvec_fp64<CPLX>(d, reinterpret_cast<const T *>(mps), y, reinterpret_cast<const T *>(envL), Rp, reinterpret_cast<const T *>(mpo),
                               ws, s));
    HEFF_TRY(dot_device<CPLX>(reinterpret_cast<const T *>(mps), y, d.size_mps(), dres, partials, s));
    T h;
    HEFF_CUDA(cudaMemcpyAsync(&h, dres, sizeof(T), cudaMemcpyDeviceToHost, s));
    HEFF_CUDA(cudaStreamSynchronize(s));
    if constexpr(CPLX) {
        result[0] = h.x;
        result[1] = h.y;
    } else {
        result[0] = h;
        result[1] = 0.0;
    }
    return HEFF_OK;
}

}  // namespace heff

using namespace heff;

extern "C" int heff_matvec_d(double *res, const double *mps, const int64_t mps_dims[3], const double *mpo, const int64_t mpo_dims[4],
                             const double *envL, const int64_t envL_dims[3], const double *envR, const int64_t envR_dims[3], void *stream) {
    return matvec_stateless<false>(res, mps, mps_dims, mpo, mpo_dims, envL, envL_dims, envR, envR_dims, (cudaStream_t)stream);
}
extern "C" int heff_matvec_z(heff_z *res, const heff_z *mps, const int64_t mps_dims[3], const heff_z *mpo, const int64_t mpo_dims[4],
                             const heff_z *envL, const int64_t envL_dims[3], const heff_z *envR, const int64_t envR_dims[3], void *stream) {
    return matvec_stateless<true>(res, mps, mps_dims, mpo, mpo_dims, envL, envL_dims, envR, envR_dims, (cudaStream_t)stream);
}
extern "C" int heff_expval_d(double *result, const double *mps, const int64_t mps_dims[3], const double *mpo, const int64_t mpo_dims[4],
                             const double *envL, const int64_t envL_dims[3], const double *envR, const int64_t envR_dims[3], void *stream) {
    return expval_stateless<false>(result, mps, mps_dims, mpo, mpo_dims, envL, envL_dims, envR, envR_dims, (cudaStream_t)stream);
}
extern "C" int heff_expval_z(double *result, const heff_z *mps, const int64_t mps_dims[3], const heff_z *mpo, const int64_t mpo_dims[4],
                             const heff_z *envL, const int64_t envL_dims[3], const heff_z *envR, const int64_t envR_dims[3], void *stream) {
    return expval_stateless<true>(result, mps, mps_dims, mpo, mpo_dims, envL, envL_dims, envR, envR_dims, (cudaStream_t)stream);
}
