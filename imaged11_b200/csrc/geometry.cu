// Detector geometry kernels: compute_gv, compute_geometry, compute_xlylzl (FP64).
//
// Streaming, bound by HBM (and by the FP64 pipe where angles are asked for).  One
// CTA of 256 threads owns a tile of 256 peaks at a time (grid-stride over tiles,
// grid = a multiple of the SM count).  The AoS
// (n,3) inputs and outputs are staged through shared memory so that every
// global access is a fully coalesced 8-byte-per-lane sweep of the tile's
// 6 KB, instead of three 24-byte-strided accesses per lane.
#include <math.h>

#include <cmath>

#include "common.cuh"
#include "tma.cuh"

namespace id11b {

struct GvParams {
    double m[9];      // chi.wedge matrix built on the host like the reference
    double t[3];      // grain translation
    double omegasign;
    double ds;        // 1 / wavelength
};

constexpr int kGeoThreads = 256;
constexpr double kRad = 3.14159265358979323846 / 180.0;
constexpr double kDeg = 180.0 / 3.14159265358979323846;

// Per-peak body of ImageD11 src/cdiffraction.c:143-167 in the reference's
// operation order (no FMA).  sin/cos come from CUDA's sincos (<= 2 ulp), the
// only difference from the reference's libm in g.
struct PeakGeo {
    double so, co, d0, d1, d2, inv, k0, k1, k2, g0, g1, g2;
};

// The angles are bound by the FP64 pipe (330 operations a peak with the library's
// arctangents, IEEE root and division: 69% of the pipe busy at 225 us for 10M peaks;
// the bytes take 147).  The two functions below take 14 operations for an
// arctangent (about 45) and 9 for 1 / sqrt (about 18).
//
// atan2 by table: with mn <= mx the two magnitudes and c = j / 64 nearest mn / mx,
//   atan(mn / mx) = atan(c) + atan(z),  z = (mn - c mx) / (mx + c mn), |z| < 2^-6.99,
// where the Taylor series of atan(z) needs four terms (the fifth is below
// 2^-59 z).  The table holds, per octant of the upper half plane, base +- atan(c)
// as two doubles, so quadrants cost no arithmetic.  z comes from one Newton step
// (2^-39) and its exact remainder goes into the sum's low part.  Against 64-bit
// mantissas over 2M detector positions: two-theta within 2.9 ulp (rms 0.61; the
// library's atan2 3.5 and 0.69, both with the root before and the degrees after),
// eta 2.6 (0.48; 2.7 and 0.49).  Magnitudes outside 2^-100 .. 2^100, zeros,
// infinities and NaN go to the library's.
constexpr int kAtanN = 64;
struct AtanTable {
    double v[4][kAtanN + 1][2];  // [|y| > |x|] + 2 [x < 0]: (value, its rounding error)
};

// atan(j / 64) times 2^100 by Euler's series, sum over n of
// 2^2n n!^2 / (2n+1)! x^(2n+1) / (1 + x^2)^(n+1), whose terms follow from one
// another by ratios of small integers (the ratio is at most 1/2)
constexpr unsigned __int128 atan_fixed(int j) {
    unsigned __int128 term = ((unsigned __int128)1 << 100) * (64 * j) / (4096 + j * j), sum = 0;
    for (int n = 0; term; n++) {
        sum += term;
        term = term * (unsigned)((2 * n + 2) * j * j) / (unsigned)((2 * n + 3) * (4096 + j * j));
    }
    return sum;
}

constexpr AtanTable make_atan_table() {
    AtanTable t{};
    const unsigned __int128 quarter = 2 * atan_fixed(kAtanN);  // pi / 2
    for (int j = 0; j <= kAtanN; j++) {
        const unsigned __int128 c = atan_fixed(j);
        for (int o = 0; o < 4; o++) {
            const unsigned __int128 v = o == 0 ? c : o == 1 ? quarter - c :
                                        o == 2 ? 2 * quarter - c : quarter + c;
            if (!v) continue;
            int sh = 0;  // v = (53 bits) 2^sh + rest
            while (v >> (sh + 53)) sh++;
            const unsigned __int128 m = (v >> sh) + ((v >> (sh - 1)) & 1);
            double a = (double)(long long)m,
                   b = (double)(long long)((unsigned long long)v - (unsigned long long)(m << sh));
            for (int k = 0; k < 100; k++) {
                if (k >= sh) a *= 0.5;
                b *= 0.5;
            }
            t.v[o][j][0] = a;
            t.v[o][j][1] = b;
        }
    }
    return t;
}
__device__ constexpr AtanTable kAtan = make_atan_table();

// The CTA's copy in shared memory: fetch, then put once the CTA's first inputs are
// asked for too, so that one latency covers both (the caller's next barrier makes the
// copy visible).  compute_geometry of 100, 20,000 and 100,000 peaks takes 2.3, 2.8 and
// 3.9 us; with the copy made first 2.8, 3.4 and 4.5, with the library's arctangents
// 2.4, 2.9 and 4.2.
struct AtanShared {
    double2 v[4][kAtanN + 1];
    static constexpr int kLen = 8 * (kAtanN + 1);
    static constexpr int kPer = (kLen + kGeoThreads - 1) / kGeoThreads;
    static __device__ __forceinline__ void fetch(double (&t)[kPer]) {
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int i = q * kGeoThreads + threadIdx.x;
            t[q] = i < kLen ? __ldg(&kAtan.v[0][0][0] + i) : 0.;
        }
    }
    __device__ __forceinline__ void put(const double (&t)[kPer]) {
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int i = q * kGeoThreads + threadIdx.x;
            if (i < kLen) (&v[0][0].x)[i] = t[q];
        }
    }
};

__device__ __forceinline__ double rcp_approx(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ double rsqrt_approx(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

// x 2^E for a normal x away from the ends of the range (integer addition)
template <int E>
__device__ __forceinline__ double times_pow2(double x) {
    return __hiloint2double(__double2hiint(x) + E * 0x00100000, __double2loint(x));
}

// the leading 24 bits of a positive double in 2^-126 .. 2^127 as a float (integer
// instructions only)
__device__ __forceinline__ float top_float(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    return __uint_as_float(__funnelshift_l(lo, hi - 0x38000000u, 3));
}

__device__ __forceinline__ double fast_atan2(double y, double x, const AtanShared& tab) {
    const int yh = __double2hiint(y), xh = __double2hiint(x);
    const long long ay = __double_as_longlong(y) & 0x7fffffffffffffffll,
                    ax = __double_as_longlong(x) & 0x7fffffffffffffffll;
    const bool swap = ay > ax;
    const double mx = __longlong_as_double(swap ? ay : ax),
                 mn = __longlong_as_double(swap ? ax : ay);
    // both within 2^-100 .. 2^100 (this leaves out zeros, infinities and NaN)
    if (__double2hiint(mn) < 0x39b00000 || __double2hiint(mx) > 0x46300000) return atan2(y, x);
    float q;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(top_float(mx)));
    const float jm = fmaf(top_float(mn) * q, (float)kAtanN, 12582912.f);  // 1.5 2^23 + j
    const int j = __float_as_int(jm) & 127;
    const unsigned cf = __float_as_uint((jm - 12582912.f) * (1.f / kAtanN));
    const double c = __hiloint2double(j ? (int)((cf >> 3) + 0x38000000u) : 0, 0);
    const int flip = swap == (xh < 0) ? 0 : (int)0x80000000;  // base - atan(c) - atan(z)
    double num = fma(-c, mx, mn);
    num = __hiloint2double(__double2hiint(num) ^ flip, __double2loint(num));
    const double den = fma(c, mn, mx);
    double r = rcp_approx(den);
    r = fma(fma(-den, r, 1.), r, r);
    const double z = num * r, z2 = z * z;  // to 2^-39: the remainder goes into the low part
    const double2 t = tab.v[(swap ? 1 : 0) + (xh < 0 ? 2 : 0)][j];
    const double p = fma(z2, fma(z2, -1. / 7., 1. / 5.), -1. / 3.);
    const double lo = fma(fma(-den, z, num), r, fma(z * z2, p, t.y));
    const double a = t.x + (z + lo);
    return __hiloint2double(__double2hiint(a) | (yh & (int)0x80000000), __double2loint(a));
}

// 1 / sqrt(x) as the two IEEE operations round it but for rare last bits: s to 2^-80
// before its rounding (Newton's steps for 1 / sqrt from the hardware's 20-bit estimate,
// then the root corrected by its exact residual, Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990), then 1 / s to 2^-80 from the
// same estimate.  A value within 2^-80 of halfway between two doubles can round the
// other way: a few of 1.6e9 arguments with these steps on a CPU, by one last place.
// 9 FP64 operations; the root and the division by themselves take about 18.
// k0 = d0 / |d| - 1 cancels near the direct beam, so a last place here is seen in g.
__device__ __forceinline__ double inv_sqrt(double x) {
    const int hi = __double2hiint(x);
    if (hi < 0x01000000 || hi > 0x7e000000) return ddiv(1., __dsqrt_rn(x));
    const double r = rsqrt_approx(x), s0 = x * r, h0 = times_pow2<-1>(r);
    const double e = fma(-s0, h0, 0.5);
    const double s1 = fma(s0, e, s0), h1 = fma(h0, e, h0);
    const double s = fma(fma(-s1, s1, x), h1, s1);
    const double y = times_pow2<1>(h1);
    return fma(fma(-s, y, 1.), y, y);
}

//
// Two specialisations give results identical to the general expression
// (apart from the sign of a zero) and are chosen on the host:
//  HAS_T = false: t == (0,0,0), so u = (+-0, +-0, 0), o = +-0 and d = xyz;
//                 taken only for a finite angle (otherwise NaN must propagate
//                 through o exactly as in the reference);
//  ROT   = false: the chi.wedge matrix is exactly the identity (wedge = chi =
//                 0) and t is finite, so M.u = u, and M^T.k = k whenever k is
//                 finite (checked per peak; 0*inf would give NaN otherwise).
template <bool HAS_T = true, bool ROT = true>
__device__ __forceinline__ void peak_geometry(const GvParams& P, double x0, double x1,
                                              double x2, double om, PeakGeo& r) {
    double ang = dmul(dmul(kRad, om), P.omegasign);
    sincos(ang, &r.so, &r.co);
    const double so = r.so, co = r.co;
    if (HAS_T || !isfinite(ang)) {
        double u0 = dsub(dmul(co, P.t[0]), dmul(so, P.t[1]));
        double u1 = dadd(dmul(so, P.t[0]), dmul(co, P.t[1]));
        double u2 = P.t[2];
        double o0 = u0, o1 = u1, o2 = u2;
        if (ROT) {
            o0 = ddot3(P.m[0], P.m[1], P.m[2], u0, u1, u2);
            o1 = ddot3(P.m[3], P.m[4], P.m[5], u0, u1, u2);
            o2 = ddot3(P.m[6], P.m[7], P.m[8], u0, u1, u2);
        }
        r.d0 = dsub(x0, o0);
        r.d1 = dsub(x1, o1);
        r.d2 = dsub(x2, o2);
    } else {
        r.d0 = x0;
        r.d1 = x1;
        r.d2 = x2;
    }
    r.inv = inv_sqrt(ddot3(r.d0, r.d1, r.d2, r.d0, r.d1, r.d2));
    r.k0 = dmul(P.ds, dsub(dmul(r.d0, r.inv), 1.));
    r.k1 = dmul(dmul(P.ds, r.d1), r.inv);
    r.k2 = dmul(dmul(P.ds, r.d2), r.inv);
    double v0, v1, v2;
    if (!ROT && isfinite(r.k0) && isfinite(r.k1) && isfinite(r.k2)) {
        v0 = r.k0;
        v1 = r.k1;
        v2 = r.k2;
    } else {
        v0 = ddot3(P.m[0], P.m[3], P.m[6], r.k0, r.k1, r.k2);
        v1 = ddot3(P.m[1], P.m[4], P.m[7], r.k0, r.k1, r.k2);
        v2 = ddot3(P.m[2], P.m[5], P.m[8], r.k0, r.k1, r.k2);
    }
    r.g0 = dadd(dmul(co, v0), dmul(so, v1));
    r.g1 = dadd(dmul(-so, v0), dmul(co, v1));
    r.g2 = v2;
}

// tth, eta, ds, g of one peak (ImageD11 src/cdiffraction.c:74-91)
__device__ __forceinline__ void geometry_out(const PeakGeo& r,
                                             const AtanShared& tab, double* o) {
    o[0] = dmul(kDeg, fast_atan2(__dsqrt_rn(dadd(dmul(r.d1, r.d1), dmul(r.d2, r.d2))), r.d0, tab));
    o[1] = dmul(kDeg, fast_atan2(-r.d1, r.d2, tab));
    o[2] = __dsqrt_rn(ddot3(r.k0, r.k1, r.k2, r.k0, r.k1, r.k2));
    o[3] = r.g0;
    o[4] = r.g1;
    o[5] = r.g2;
}

// MODE 0: gv (n,3); MODE 1: geometry out (n,6)
template <int MODE>
__global__ void __launch_bounds__(kGeoThreads)
k_geometry(const double* __restrict__ xyz, const double* __restrict__ omega, GvParams P,
           double* __restrict__ out, float4* __restrict__ g4, int64_t n) {
    constexpr int OUTW = MODE == 0 ? 3 : 6;
    __shared__ AtanShared s_tab;  // (MODE 0 has no angles and no table)
    __shared__ double s_in[3 * kGeoThreads];
    __shared__ double s_out[OUTW * kGeoThreads];
    const int tid = threadIdx.x;
    if (MODE == 1) {
        double tab[AtanShared::kPer];
        AtanShared::fetch(tab);
        // the first tile's lines (16 doubles each: xyz's, then omega's)
        constexpr int kLines = 3 * kGeoThreads / 16;
        const bool x = tid < kLines;
        const int64_t at = (int64_t)blockIdx.x * kGeoThreads * (x ? 3 : 1) +
                           16 * (x ? tid : tid - kLines);
        if (tid < kLines + kGeoThreads / 16 && at < (x ? 3 * n : n))
            asm volatile("prefetch.global.L1 [%0];" ::"l"((x ? xyz : omega) + at));
        s_tab.put(tab);
    }
    for (int64_t base = (int64_t)blockIdx.x * kGeoThreads; base < n;
         base += (int64_t)gridDim.x * kGeoThreads) {
        const int cnt = (int)min((int64_t)kGeoThreads, n - base);
        const double* src = xyz + 3 * base;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            int e = tid + j * kGeoThreads;
            if (e < 3 * cnt) s_in[e] = __ldcs(src + e);
        }
        double om = tid < cnt ? __ldcs(omega + base + tid) : 0.;
        __syncthreads();
        if (tid < cnt) {
            PeakGeo r;
            peak_geometry(P, s_in[3 * tid], s_in[3 * tid + 1], s_in[3 * tid + 2], om, r);
            if (MODE == 0) {
                s_out[3 * tid] = r.g0;
                s_out[3 * tid + 1] = r.g1;
                s_out[3 * tid + 2] = r.g2;
                if (g4)
                    g4[base + tid] = make_float4((float)r.g0, (float)r.g1, (float)r.g2, 0.f);
            } else {
                geometry_out(r, s_tab, s_out + 6 * tid);
            }
        }
        __syncthreads();
        double* dst = out + OUTW * base;
#pragma unroll
        for (int j = 0; j < OUTW; j++) {
            int e = tid + j * kGeoThreads;
            if (e < OUTW * cnt) __stcs(dst + e, s_out[e]);
        }
        __syncthreads();
    }
}

// Pipelined variant for 16-byte-aligned inputs: a persistent CTA walks its
// tiles (blockIdx.x, +gridDim.x, ...) with a ring of S stages of 1-D TMA bulk
// copies (xyz 6 KB + omega 2 KB per tile) completed on mbarriers, so the loads
// of the next S - 1 tiles are in flight while the current one is computed and
// stored.  The final partial tile, whose byte counts need not be multiples of
// 16, is read with ordinary loads.  Bounded waits: on a timeout the CTA stops
// and counts the event in g_geo_timeouts.
__device__ unsigned int g_geo_timeouts = 0;

template <int MODE, bool HAS_T = true, bool ROT = true>
__global__ void __launch_bounds__(kGeoThreads, 4)
k_geometry_tma(const double* __restrict__ xyz, const double* __restrict__ omega, GvParams P,
               double* __restrict__ out, float4* __restrict__ g4, int64_t n) {
    constexpr int OUTW = MODE == 0 ? 3 : 6;
    constexpr int S = MODE == 0 ? 4 : 3;  // (38 KB in all; MODE 1, with the table, 40)
    __shared__ AtanShared s_tab;  // (MODE 0 has no angles and no table)
    double tab[AtanShared::kPer];
    if (MODE == 1) AtanShared::fetch(tab);
    __shared__ __align__(128) double s_x[S][3 * kGeoThreads];
    __shared__ __align__(128) double s_w[S][kGeoThreads];
    __shared__ __align__(16) double s_out[OUTW * kGeoThreads];
    __shared__ __align__(8) uint64_t s_bar[S];
    const int tid = threadIdx.x;
    const int64_t ntiles = (n + kGeoThreads - 1) / kGeoThreads;
    const int64_t nfull = n / kGeoThreads;
    auto issue = [&](int stage, int64_t t) {
        mbar_arrive_expect_tx(&s_bar[stage], (3 + 1) * kGeoThreads * sizeof(double));
        tma_load_1d(s_x[stage], xyz + 3 * t * kGeoThreads, 3 * kGeoThreads * sizeof(double),
                    &s_bar[stage]);
        tma_load_1d(s_w[stage], omega + t * kGeoThreads, kGeoThreads * sizeof(double),
                    &s_bar[stage]);
    };
    if (tid == 0) {
        for (int s = 0; s < S; s++) mbar_init(&s_bar[s], 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (tid == 0)
        for (int s = 0; s < S; s++) {
            int64_t t = blockIdx.x + (int64_t)s * gridDim.x;
            if (t < nfull) issue(s, t);
        }
    if (MODE == 1) {
        s_tab.put(tab);
        __syncthreads();
    }
    for (int64_t i = 0;; i++) {
        const int64_t t = blockIdx.x + i * gridDim.x;
        if (t >= ntiles) break;
        const int stage = (int)(i % S);
        const int64_t base = t * kGeoThreads;
        const int cnt = (int)min((int64_t)kGeoThreads, n - base);
        double x0 = 0., x1 = 0., x2 = 0., om = 0.;
        if (t < nfull) {
            if (!__syncthreads_and(mbar_wait_bounded(&s_bar[stage], (uint32_t)((i / S) & 1)))) {
                if (tid == 0) {
                    atomicAdd(&g_geo_timeouts, 1u);
                    for (int64_t j = i; j < i + S; j++)  // copies still in flight
                        if (blockIdx.x + j * gridDim.x < nfull)
                            mbar_wait_bounded(&s_bar[j % S], (uint32_t)((j / S) & 1), 1u << 16);
                }
                return;
            }
            x0 = s_x[stage][3 * tid];
            x1 = s_x[stage][3 * tid + 1];
            x2 = s_x[stage][3 * tid + 2];
            om = s_w[stage][tid];
        } else if (tid < cnt) {  // final partial tile
            x0 = xyz[3 * (base + tid)];
            x1 = xyz[3 * (base + tid) + 1];
            x2 = xyz[3 * (base + tid) + 2];
            om = omega[base + tid];
        }
        if (tid < cnt) {
            PeakGeo r;
            peak_geometry<HAS_T, ROT>(P, x0, x1, x2, om, r);
            if (MODE == 0) {
                s_out[3 * tid] = r.g0;
                s_out[3 * tid + 1] = r.g1;
                s_out[3 * tid + 2] = r.g2;
                if (g4) g4[base + tid] = make_float4((float)r.g0, (float)r.g1, (float)r.g2, 0.f);
            } else {
                geometry_out(r, s_tab, s_out + 6 * tid);
            }
        }
        __syncthreads();  // stage consumed by every lane; s_out complete
        if (tid == 0) {
            const int64_t tn = blockIdx.x + (i + S) * gridDim.x;
            if (tn < nfull) {
                fence_proxy_async_smem();
                issue(stage, tn);
            }
        }
        double* dst = out + OUTW * base;
#pragma unroll
        for (int j = 0; j < OUTW; j++) {
            int e = tid + j * kGeoThreads;
            if (e < OUTW * cnt) dst[e] = s_out[e];
        }
        __syncthreads();  // s_out free for the next tile
    }
}

// ImageD11 src/cdiffraction.c:190-224: xlylzl_j = r[3j+1]*v1 + r[3j+2]*v2 + dist_j
struct XyzParams {
    double p[4];
    double r[9];
    double dist[3];
};

__global__ void __launch_bounds__(kGeoThreads)
k_xlylzl(const double* __restrict__ s, const double* __restrict__ f, XyzParams P,
         double* __restrict__ out, int64_t n) {
    __shared__ double s_out[3 * kGeoThreads];
    const int tid = threadIdx.x;
    for (int64_t base = (int64_t)blockIdx.x * kGeoThreads; base < n;
         base += (int64_t)gridDim.x * kGeoThreads) {
        const int cnt = (int)min((int64_t)kGeoThreads, n - base);
        if (tid < cnt) {
            double v1 = dmul(dsub(__ldcs(f + base + tid), P.p[1]), P.p[3]);
            double v2 = dmul(dsub(__ldcs(s + base + tid), P.p[0]), P.p[2]);
#pragma unroll
            for (int j = 0; j < 3; j++)
                s_out[3 * tid + j] =
                    dadd(dadd(dmul(P.r[3 * j + 1], v1), dmul(P.r[3 * j + 2], v2)), P.dist[j]);
        }
        __syncthreads();
        double* dst = out + 3 * base;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            int e = tid + j * kGeoThreads;
            if (e < 3 * cnt) __stcs(dst + e, s_out[e]);
        }
        __syncthreads();
    }
}

// Detector position -> lab position -> geometry in one pass (the two calls of
// columnfile.updateGeometry's fast path, ImageD11/columnfile.py:497-504:
// Ctransform.sf2xyz = compute_xlylzl, then xyz2geometry = compute_geometry).
// The lab positions never leave registers unless asked for, and each value is
// produced by the same operations as the two separate kernels, so the results
// are identical to calling them in turn.  sc, fc, omega are read once with
// the next tile's loads issued before the current tile is computed.
//
// A warp owns tiles of 32 peaks: its outputs go through its own part of shared
// memory, so no warp waits for another.  10M peaks with the lab positions: 225 us with
// the library's arctangents and a CTA's 256 peaks behind two barriers, 174 now (5.5
// TB/s); two waves of CTAs, since one ended unevenly (186).
template <bool XYZ, bool G4>
__global__ void __launch_bounds__(kGeoThreads, 4)
k_update_geometry(const double* __restrict__ sc, const double* __restrict__ fc,
                  const double* __restrict__ omega, XyzParams X, GvParams P,
                  double* __restrict__ xyz, double* __restrict__ out, float4* __restrict__ g4,
                  int64_t n) {
    __shared__ AtanShared s_tab;
    __shared__ double s_xyz[XYZ ? 3 * kGeoThreads : 1];
    __shared__ double s_out[6 * kGeoThreads];
    double tab[AtanShared::kPer];
    AtanShared::fetch(tab);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* const wx = s_xyz + (XYZ ? 96 * warp : 0);
    double* const wo = s_out + 192 * warp;
    const int64_t step = (int64_t)gridDim.x * kGeoThreads;
    double sn = 0., fn = 0., on = 0.;
    auto load = [&](int64_t base) {
        const int64_t k = base + lane;
        if (k < n) {
            sn = __ldcs(sc + k);
            fn = __ldcs(fc + k);
            on = __ldcs(omega + k);
        }
    };
    int64_t base = (int64_t)blockIdx.x * kGeoThreads + 32 * warp;
    load(base);
    s_tab.put(tab);
    __syncthreads();
    for (; base < n; base += step) {
        const double s = sn, f = fn, om = on;
        load(base + step);
        const int cnt = (int)min((int64_t)32, n - base);
        if (lane < cnt) {
            const double v1 = dmul(dsub(f, X.p[1]), X.p[3]);
            const double v2 = dmul(dsub(s, X.p[0]), X.p[2]);
            double x[3];
#pragma unroll
            for (int j = 0; j < 3; j++) {
                x[j] = dadd(dadd(dmul(X.r[3 * j + 1], v1), dmul(X.r[3 * j + 2], v2)), X.dist[j]);
                if (XYZ) wx[3 * lane + j] = x[j];
            }
            PeakGeo r;
            peak_geometry(P, x[0], x[1], x[2], om, r);
            geometry_out(r, s_tab, wo + 6 * lane);
            if (G4) g4[base + lane] = make_float4((float)r.g0, (float)r.g1, (float)r.g2, 0.f);
        }
        __syncwarp();
        if (XYZ) {
            double* dx = xyz + 3 * base;
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const int e = lane + 32 * j;
                if (e < 3 * cnt) __stcs(dx + e, wx[e]);
            }
        }
        double* dst = out + 6 * base;
#pragma unroll
        for (int j = 0; j < 6; j++) {
            const int e = lane + 32 * j;
            if (e < 6 * cnt) __stcs(dst + e, wo[e]);
        }
        __syncwarp();
    }
}

// Chi.wedge matrix exactly as ImageD11 src/cdiffraction.c:117-142 (host libm,
// the reference's own sin/cos; the macro RAD expands to (x*pi)/180 here).
static void wedgechi_host(double wedge, double chi, double m[9]) {
    const double pi = 3.14159265358979323846;
    double sw = sin(wedge * pi / 180.0), cw = cos(wedge * pi / 180.0);
    double sc = sin(chi * pi / 180.0), cc = cos(chi * pi / 180.0);
    double w[9] = {cw, 0.0, -sw, 0., 1.0, 0., sw, 0.0, cw};
    double c[9] = {1., 0.0, 0., 0., cc, -sc, 0., sc, cc};
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            volatile double a = c[j] * w[3 * i];
            volatile double b = c[3 + j] * w[3 * i + 1];
            volatile double d = c[6 + j] * w[3 * i + 2];
            volatile double ab = a + b;
            m[3 * i + j] = ab + d;
        }
}

static bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

static int geo_grid_tma(int64_t n) {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    int64_t tiles = (n + kGeoThreads - 1) / kGeoThreads;
    int64_t g = (int64_t)sms * 4;  // 4 persistent CTAs per SM (shared memory <= 44 KB each)
    return (int)(tiles < g ? (tiles > 0 ? tiles : 1) : g);
}

static int geo_grid(int64_t n) {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    int64_t tiles = (n + kGeoThreads - 1) / kGeoThreads;
    int64_t g = (int64_t)sms * 8;  // two waves of the kernels with 4 CTAs per SM
    return (int)(tiles < g ? (tiles > 0 ? tiles : 1) : g);
}

}  // namespace id11b

using namespace id11b;

static GvParams make_gv_params(double omegasign, double wvln, double wedge, double chi,
                               const double* t) {
    GvParams P;
    wedgechi_host(wedge, chi, P.m);
    for (int i = 0; i < 3; i++) P.t[i] = t[i];
    P.omegasign = omegasign;
    volatile double one = 1.;
    P.ds = one / wvln;
    return P;
}

extern "C" int id11b_dev_compute_gv(const double* xlylzl, const double* omega,
                                    double omegasign, double wvln, double wedge, double chi,
                                    const double* t_host, double* gv, float* g4, int64_t n,
                                    void* stream) {
    if (n < 0 || !t_host) return ID11B_ERR_ARG;
    if (n == 0) return ID11B_OK;
    if (!xlylzl || !omega || !gv) return ID11B_ERR_ARG;
    if (g4 && ((uintptr_t)g4 & 15)) return ID11B_ERR_ALIGN;
    GvParams P = make_gv_params(omegasign, wvln, wedge, chi, t_host);
    const bool has_t = !(t_host[0] == 0. && t_host[1] == 0. && t_host[2] == 0.);
    bool rot = !(std::isfinite(t_host[0]) && std::isfinite(t_host[1]) && std::isfinite(t_host[2]));
    for (int i = 0; i < 9; i++) rot = rot || P.m[i] != (i % 4 == 0 ? 1. : 0.);
    cudaStream_t st = (cudaStream_t)stream;
    const int grid = geo_grid_tma(n);
    if (aligned16(xlylzl) && aligned16(omega)) {
        if (has_t && rot)
            k_geometry_tma<0, true, true><<<grid, kGeoThreads, 0, st>>>(xlylzl, omega, P, gv,
                                                                        (float4*)g4, n);
        else if (has_t)
            k_geometry_tma<0, true, false><<<grid, kGeoThreads, 0, st>>>(xlylzl, omega, P, gv,
                                                                         (float4*)g4, n);
        else if (rot)
            k_geometry_tma<0, false, true><<<grid, kGeoThreads, 0, st>>>(xlylzl, omega, P, gv,
                                                                         (float4*)g4, n);
        else
            k_geometry_tma<0, false, false><<<grid, kGeoThreads, 0, st>>>(xlylzl, omega, P, gv,
                                                                          (float4*)g4, n);
    } else
        k_geometry<0><<<geo_grid(n), kGeoThreads, 0, (cudaStream_t)stream>>>(
            xlylzl, omega, P, gv, (float4*)g4, n);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_compute_geometry(const double* xlylzl, const double* omega,
                                          double omegasign, double wvln, double wedge,
                                          double chi, const double* t_host, double* out,
                                          int64_t n, void* stream) {
    if (n < 0 || !t_host) return ID11B_ERR_ARG;
    if (n == 0) return ID11B_OK;
    if (!xlylzl || !omega || !out) return ID11B_ERR_ARG;
    GvParams P = make_gv_params(omegasign, wvln, wedge, chi, t_host);
    if (aligned16(xlylzl) && aligned16(omega))
        k_geometry_tma<1><<<geo_grid_tma(n), kGeoThreads, 0, (cudaStream_t)stream>>>(
            xlylzl, omega, P, out, nullptr, n);
    else
        k_geometry<1><<<geo_grid(n), kGeoThreads, 0, (cudaStream_t)stream>>>(xlylzl, omega, P,
                                                                             out, nullptr, n);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_compute_xlylzl(const double* s, const double* f,
                                        const double* p_host, const double* r_host,
                                        const double* dist_host, double* xlylzl, int64_t n,
                                        void* stream) {
    if (n < 0 || !p_host || !r_host || !dist_host) return ID11B_ERR_ARG;
    if (n == 0) return ID11B_OK;
    if (!s || !f || !xlylzl) return ID11B_ERR_ARG;
    XyzParams P;
    for (int i = 0; i < 4; i++) P.p[i] = p_host[i];
    for (int i = 0; i < 9; i++) P.r[i] = r_host[i];
    for (int i = 0; i < 3; i++) P.dist[i] = dist_host[i];
    k_xlylzl<<<geo_grid(n), kGeoThreads, 0, (cudaStream_t)stream>>>(s, f, P, xlylzl, n);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_update_geometry(const double* sc, const double* fc, const double* omega,
                                         const double* p_host, const double* r_host,
                                         const double* dist_host, double omegasign, double wvln,
                                         double wedge, double chi, const double* t_host,
                                         double* xlylzl, double* out, float* g4, int64_t n,
                                         void* stream) {
    if (n < 0 || !p_host || !r_host || !dist_host || !t_host) return ID11B_ERR_ARG;
    if (n == 0) return ID11B_OK;
    if (!sc || !fc || !omega || !out) return ID11B_ERR_ARG;
    if (g4 && ((uintptr_t)g4 & 15)) return ID11B_ERR_ALIGN;
    XyzParams X;
    for (int i = 0; i < 4; i++) X.p[i] = p_host[i];
    for (int i = 0; i < 9; i++) X.r[i] = r_host[i];
    for (int i = 0; i < 3; i++) X.dist[i] = dist_host[i];
    GvParams P = make_gv_params(omegasign, wvln, wedge, chi, t_host);
    cudaStream_t st = (cudaStream_t)stream;
    const int grid = geo_grid(n);
    if (xlylzl && g4)
        k_update_geometry<true, true><<<grid, kGeoThreads, 0, st>>>(sc, fc, omega, X, P, xlylzl,
                                                                    out, (float4*)g4, n);
    else if (xlylzl)
        k_update_geometry<true, false><<<grid, kGeoThreads, 0, st>>>(sc, fc, omega, X, P, xlylzl,
                                                                     out, nullptr, n);
    else if (g4)
        k_update_geometry<false, true><<<grid, kGeoThreads, 0, st>>>(sc, fc, omega, X, P, nullptr,
                                                                     out, (float4*)g4, n);
    else
        k_update_geometry<false, false><<<grid, kGeoThreads, 0, st>>>(sc, fc, omega, X, P,
                                                                      nullptr, out, nullptr, n);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}
