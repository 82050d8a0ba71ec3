// Per-grain translation refinement: the objective of
// ImageD11/refinegrains.py refinepositions (:636-660) / gof (:517-560),
// minimised by damped Gauss-Newton for every grain at once instead of a
// Nelder-Mead simplex per grain.
//
// For grain G with peaks k (lab positions x_k, omega_k) and the UBI it was
// read with, U0, the reference's gof at translation t is built by
// refinegrains.refine (:459-498): g_k(t) from compute_gv (ImageD11
// src/cdiffraction.c:112-168), one score_and_refine from U0 at tol (the
// least-squares UBI U1 of the peaks with drlv2 < tol^2, hkl = round(U0.g)),
// then a second score_and_refine at U1 whose mean drlv2 is the objective:
//   cost(t) = sum over peaks with drlv2 < tol^2 of |U1.g_k - round(U1.g_k)|^2.
// Each iteration makes the same two passes over the grain's peaks: the first
// sums R = sum g h^T and H = sum h h^T and solves U1 = (R H^-1)^-1; the
// second takes the cost at U1 and, with U1 and the rounded hkl held for the
// step, the Jacobian of r_k = U1.g_k(t) - hkl,
//   dr/dt = U1 . B . M^T . (ds/|d|)(I - n n^T) . (-M . A),
// A = dR_omega/dt (the omega rotation of t), B the omega rotation of g,
// d = x - M.A.t, n = d/|d| (forward mode, three tangents per peak; the
// adjoint's reverse pass gives J^T r but not the J^T J a Gauss-Newton step
// needs).  Holding U1 is exact for the gradient: at the least-squares U1 the
// derivative of the cost through U1 vanishes.  The sums J^T J, J^T r and the
// cost are reduced in a fixed order and a Levenberg-Marquardt step is taken;
// a step that raises the cost is undone and the damping raised.  One CTA per
// grain, every iteration in one launch; sin and cos of a peak's omega, and the
// 1 / |d| that the second pass shares with the first, are kept in shared memory
// by the thread that owns the peak.
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace id11b {
namespace trans {

constexpr int kTT = 64;  // threads per grain
constexpr int kResident = 4;  // CTAs per SM at most (226 registers)
// peaks per thread kept in shared memory (three doubles each: 24 KB a CTA); the
// peaks of a larger grain beyond 64 x 16 are computed in each pass
constexpr int kKeep = 16;
constexpr double kRad = 3.14159265358979323846 / 180.0;

struct Geo {
    double m[9];  // chi.wedge
    double omegasign, ds;
    double tol2;
};

// sums of one peak: J^T J (6, upper), J^T r (3), cost, n
struct Acc {
    double a[11];
};

// g of one peak at translation t, with what its tangents need; so and co (and inv
// when HAVE) given.  Near the minimum a step is taken or refused by the last bits
// of the cost, so the passes compute g each in its own way, as they always did:
// taking the first pass's g in the second moves t by 1e-8 of itself.
struct PeakG {
    double so, co, n0, n1, n2, inv, g[3];
};

template <bool HAVE>
__device__ __forceinline__ void peak_g(const Geo& P, const double t[3], double x0, double x1,
                                       double x2, PeakG& q) {
    const double* M = P.m;
    const double so = q.so, co = q.co;
    // o = M.A.t, A = [[co,-so,0],[so,co,0],[0,0,1]]
    const double at0 = co * t[0] - so * t[1], at1 = so * t[0] + co * t[1], at2 = t[2];
    const double d0 = x0 - (M[0] * at0 + M[1] * at1 + M[2] * at2);
    const double d1 = x1 - (M[3] * at0 + M[4] * at1 + M[5] * at2);
    const double d2 = x2 - (M[6] * at0 + M[7] * at1 + M[8] * at2);
    if (!HAVE) q.inv = 1.0 / sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    q.n0 = d0 * q.inv;
    q.n1 = d1 * q.inv;
    q.n2 = d2 * q.inv;
    const double k0 = P.ds * (q.n0 - 1.0), k1 = P.ds * q.n1, k2 = P.ds * q.n2;
    const double v0 = M[0] * k0 + M[3] * k1 + M[6] * k2;
    const double v1 = M[1] * k0 + M[4] * k1 + M[7] * k2;
    const double v2 = M[2] * k0 + M[5] * k1 + M[8] * k2;
    q.g[0] = co * v0 + so * v1;
    q.g[1] = -so * v0 + co * v1;
    q.g[2] = v2;
}

// first pass: R (9, R[i][j] = sum h_j g_i) and H (6, upper) of the peaks
// with drlv2(u0) < tol^2, as score_and_refine sums them
__device__ __forceinline__ void refit_terms(const Geo& P, const double u[9], const PeakG& q,
                                            double* a) {
    double ih[3], r[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double h = u[3 * i] * q.g[0] + u[3 * i + 1] * q.g[1] + u[3 * i + 2] * q.g[2];
        ih[i] = rint(h);
        r[i] = h - ih[i];
    }
    const double s = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    if (!(s < P.tol2)) return;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) a[3 * i + j] += ih[j] * q.g[i];
    a[9] += ih[0] * ih[0];
    a[10] += ih[0] * ih[1];
    a[11] += ih[0] * ih[2];
    a[12] += ih[1] * ih[1];
    a[13] += ih[1] * ih[2];
    a[14] += ih[2] * ih[2];
}

// second pass: cost and Gauss-Newton sums at u
__device__ __forceinline__ void peak_terms(const Geo& P, const double u[9], const PeakG& q,
                                           Acc& acc) {
    const double* M = P.m;
    const double so = q.so, co = q.co, n0 = q.n0, n1 = q.n1, n2 = q.n2, inv = q.inv;
    double r[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double h = u[3 * i] * q.g[0] + u[3 * i + 1] * q.g[1] + u[3 * i + 2] * q.g[2];
        r[i] = h - rint(h);
    }
    const double s = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    if (!(s < P.tol2)) return;
    // columns j of dd/dt = -M.A e_j
    const double A[3][3] = {{co, -so, 0.}, {so, co, 0.}, {0., 0., 1.}};
    double J[3][3];  // J[i][j] = dr_i / dt_j
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const double a0 = A[0][j], a1 = A[1][j], a2 = A[2][j];
        const double e0 = -(M[0] * a0 + M[1] * a1 + M[2] * a2);
        const double e1 = -(M[3] * a0 + M[4] * a1 + M[5] * a2);
        const double e2 = -(M[6] * a0 + M[7] * a1 + M[8] * a2);
        // dk = ds * inv * (e - n (n.e))
        const double ne = n0 * e0 + n1 * e1 + n2 * e2;
        const double q0 = P.ds * inv * (e0 - n0 * ne), q1 = P.ds * inv * (e1 - n1 * ne),
                     q2 = P.ds * inv * (e2 - n2 * ne);
        const double w0 = M[0] * q0 + M[3] * q1 + M[6] * q2;
        const double w1 = M[1] * q0 + M[4] * q1 + M[7] * q2;
        const double w2 = M[2] * q0 + M[5] * q1 + M[8] * q2;
        const double dg0 = co * w0 + so * w1, dg1 = -so * w0 + co * w1, dg2 = w2;
#pragma unroll
        for (int i = 0; i < 3; i++) J[i][j] = u[3 * i] * dg0 + u[3 * i + 1] * dg1 + u[3 * i + 2] * dg2;
    }
    int k = 0;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = a; b < 3; b++) {
            acc.a[k++] += J[0][a] * J[0][b] + J[1][a] * J[1][b] + J[2][a] * J[2][b];
        }
#pragma unroll
    for (int a = 0; a < 3; a++) acc.a[6 + a] += J[0][a] * r[0] + J[1][a] * r[1] + J[2][a] * r[2];
    acc.a[9] += s;
    acc.a[10] += 1.0;
}

// (H + lambda diag H) x = -b for a symmetric 3x3 H (upper: h00 h01 h02 h11 h12 h22)
__device__ __forceinline__ bool solve3(const double h[6], const double b[3], double lam,
                                       double x[3]) {
    const double a00 = h[0] * (1. + lam), a01 = h[1], a02 = h[2];
    const double a11 = h[3] * (1. + lam), a12 = h[4], a22 = h[5] * (1. + lam);
    const double c00 = a11 * a22 - a12 * a12, c01 = a02 * a12 - a01 * a22,
                 c02 = a01 * a12 - a02 * a11;
    const double det = a00 * c00 + a01 * c01 + a02 * c02;
    if (!(fabs(det) > 0.) || !isfinite(det)) return false;
    const double c11 = a00 * a22 - a02 * a02, c12 = a01 * a02 - a00 * a12,
                 c22 = a00 * a11 - a01 * a01;
    const double id = -1.0 / det;
    x[0] = id * (c00 * b[0] + c01 * b[1] + c02 * b[2]);
    x[1] = id * (c01 * b[0] + c11 * b[1] + c12 * b[2]);
    x[2] = id * (c02 * b[0] + c12 * b[1] + c22 * b[2]);
    return isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]);
}

// U1 = (R H^-1)^-1 from the first pass's sums (a: lane q < 15 holds the q-th), one
// element per lane, by one warp; u0 when H or R H^-1 is singular, as
// score_and_refine leaves its UBI.  m: nine doubles of scratch in shared memory.
__device__ __forceinline__ double refit_ubi(double a, double u0, double* m, int lane) {
    const int e = lane < 9 ? lane : 0, i = e / 3, j = e - 3 * i;
    const double h = __shfl_sync(0xffffffffu, a, 9 + (i + j + (min(i, j) > 0)));
    if (lane < 9) m[e] = h;
    __syncwarp();
    const double det = det3_exact(m);
    const double hi = det != 0. ? inv3_elem(m, det, e) : 0.;
    double r[3], c[3];
#pragma unroll
    for (int l = 0; l < 3; l++) {
        r[l] = __shfl_sync(0xffffffffu, a, 3 * i + l);
        c[l] = __shfl_sync(0xffffffffu, hi, 3 * l + j);
    }
    __syncwarp();
    if (lane < 9) m[e] = r[0] * c[0] + r[1] * c[1] + r[2] * c[2];
    __syncwarp();
    const double det2 = det3_exact(m);
    return det != 0. && det2 != 0. ? inv3_elem(m, det2, e) : u0;
}

// Bound: the FP64 pipe of the SMs that hold four grains (500 grains are 3.4 CTAs
// per SM), at two warps per scheduler.  500 grains of 420 .. 560 peaks, 30
// iterations: 0.30 ms; 0.43 with sin, cos and 1 / |d| taken in every pass, full
// butterflies and one thread's 3x3 solves.  Two or four peaks at a time: 0.32, 0.35.
// The peaks beyond the kept ones have loops of their own: in one loop with a branch
// 10 grains of 14,700 peaks, 10 iterations, took 4.2 ms instead of 3.45.
__global__ void __launch_bounds__(kTT)
k_refine_translations(const double* __restrict__ xyz, const double* __restrict__ omega,
                      const int64_t* __restrict__ offsets, int32_t ngrains,
                      const double* __restrict__ ubis, double* __restrict__ tr, Geo P, int iters,
                      double* __restrict__ cost_out, int32_t* __restrict__ npk_out,
                      double* __restrict__ ubi_out) {
    __shared__ double s_red[kTT / 32][15];
    __shared__ double s_t[3], s_u[9], s_m[9];
    extern __shared__ double s_keep[];  // [field][peak of the thread][thread]
    const int gi = blockIdx.x;
    if (gi >= ngrains) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t p0 = offsets[gi];
    const int64_t np = offsets[gi + 1] - p0;
    double* const keep = s_keep + tid;
    constexpr int kF = kKeep * kTT;  // doubles per field
    auto angles = [&](int64_t k, PeakG& q) {
        sincos(kRad * omega[p0 + k] * P.omegasign, &q.so, &q.co);
    };
    // the thread's peaks that are kept, and their positions
    const int kept = (int)min((int64_t)kKeep, (np - tid + kTT - 1) / kTT);
    const double* const mine = xyz + 3 * (p0 + tid);
    for (int i = 0; i < kept; i++) {
        PeakG q;
        angles(tid + kTT * i, q);
        keep[i * kTT] = q.so;
        keep[kF + i * kTT] = q.co;
    }
    double u0[9];
#pragma unroll
    for (int e = 0; e < 9; e++) u0[e] = ubis[9 * gi + e];
    const double u0e = ubis[9 * gi + (lane < 9 ? lane : 0)];
    double tacc[3] = {tr[3 * gi], tr[3 * gi + 1], tr[3 * gi + 2]};
    double hacc[6] = {0, 0, 0, 0, 0, 0}, bacc[3] = {0, 0, 0}, cacc = 0., nacc = 0.;
    double uacc[9];
#pragma unroll
    for (int e = 0; e < 9; e++) uacc[e] = u0[e];
    double lam = 1e-3;
    if (tid == 0) {
        s_t[0] = tacc[0];
        s_t[1] = tacc[1];
        s_t[2] = tacc[2];
    }
    __syncthreads();
    for (int it = 0; it <= iters; it++) {
        const double t[3] = {s_t[0], s_t[1], s_t[2]};
        // pass 1: least-squares UBI from u0 at t
        double a[15];
#pragma unroll
        for (int q = 0; q < 15; q++) a[q] = 0.;
        for (int i = 0; i < kept; i++) {
            const double* x = mine + 3 * kTT * i;
            PeakG q;
            q.so = keep[i * kTT];
            q.co = keep[kF + i * kTT];
            peak_g<false>(P, t, x[0], x[1], x[2], q);
            keep[2 * kF + i * kTT] = q.inv;
            refit_terms(P, u0, q, a);
        }
        for (int64_t k = tid + kKeep * kTT; k < np; k += kTT) {
            const double* x = xyz + 3 * (p0 + k);
            const double x0 = x[0], x1 = x[1], x2 = x[2];
            PeakG q;
            angles(k, q);
            peak_g<false>(P, t, x0, x1, x2, q);
            refit_terms(P, u0, q, a);
        }
        {
            const int f = slot_of<15>(lane);
            const double v = ScatterSum<15, 16>::run(a, lane);
            if (f >= 0) s_red[wid][f] = v;
        }
        __syncthreads();
        if (wid == 0) {
            double v = 0.;
            if (lane < 15)
                for (int w = 0; w < kTT / 32; w++) v += s_red[w][lane];  // fixed order
            v = refit_ubi(v, u0e, s_m, lane);
            if (lane < 9) s_u[lane] = v;
        }
        __syncthreads();
        double u1[9];
#pragma unroll
        for (int e = 0; e < 9; e++) u1[e] = s_u[e];
        // pass 2: cost and Gauss-Newton sums at u1
        Acc acc;
#pragma unroll
        for (int q = 0; q < 11; q++) acc.a[q] = 0.;
        for (int i = 0; i < kept; i++) {
            PeakG q;
            const double* x = mine + 3 * kTT * i;
            q.so = keep[i * kTT];
            q.co = keep[kF + i * kTT];
            q.inv = keep[2 * kF + i * kTT];
            peak_g<true>(P, t, x[0], x[1], x[2], q);
            peak_terms(P, u1, q, acc);
        }
        for (int64_t k = tid + kKeep * kTT; k < np; k += kTT) {
            const double* x = xyz + 3 * (p0 + k);
            const double x0 = x[0], x1 = x[1], x2 = x[2];
            PeakG q;
            angles(k, q);
            peak_g<false>(P, t, x0, x1, x2, q);
            peak_terms(P, u1, q, acc);
        }
        {
            const int f = slot_of<11>(lane);
            const double v = ScatterSum<11, 16>::run(acc.a, lane);
            if (f >= 0) s_red[wid][f] = v;
        }
        __syncthreads();
        if (tid == 0) {
            double r[11];
            for (int q = 0; q < 11; q++) {
                r[q] = 0.;
                for (int w = 0; w < kTT / 32; w++) r[q] += s_red[w][q];  // fixed order
            }
            if (it == 0 || r[9] < cacc) {  // accept t (or the start point)
                for (int q = 0; q < 6; q++) hacc[q] = r[q];
                for (int q = 0; q < 3; q++) {
                    bacc[q] = r[6 + q];
                    tacc[q] = t[q];
                }
                for (int e = 0; e < 9; e++) uacc[e] = u1[e];
                cacc = r[9];
                nacc = r[10];
                if (it) lam = fmax(lam * 0.3, 1e-9);
            } else {
                lam = fmin(lam * 10., 1e9);
            }
            double x[3] = {0., 0., 0.};
            if (it < iters && nacc >= 3. && solve3(hacc, bacc, lam, x)) {
                s_t[0] = tacc[0] + x[0];
                s_t[1] = tacc[1] + x[1];
                s_t[2] = tacc[2] + x[2];
            } else {
                s_t[0] = tacc[0];
                s_t[1] = tacc[1];
                s_t[2] = tacc[2];
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        tr[3 * gi] = tacc[0];
        tr[3 * gi + 1] = tacc[1];
        tr[3 * gi + 2] = tacc[2];
        if (cost_out) cost_out[gi] = cacc;
        if (npk_out) npk_out[gi] = (int32_t)nacc;
        if (ubi_out)
            for (int e = 0; e < 9; e++) ubi_out[9 * gi + e] = uacc[e];
    }
}

}  // namespace trans
}  // namespace id11b

using namespace id11b::trans;

// chi.wedge as the reference builds it (src/cdiffraction.c:117-142)
static void wedgechi(double wedge, double chi, double m[9]) {
    const double pi = 3.14159265358979323846;
    double sw = sin(wedge * pi / 180.0), cw = cos(wedge * pi / 180.0);
    double sc = sin(chi * pi / 180.0), cc = cos(chi * pi / 180.0);
    double w[9] = {cw, 0.0, -sw, 0., 1.0, 0., sw, 0.0, cw};
    double c[9] = {1., 0.0, 0., 0., cc, -sc, 0., sc, cc};
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++)
            m[3 * i + j] = c[j] * w[3 * i] + c[3 + j] * w[3 * i + 1] + c[6 + j] * w[3 * i + 2];
}

extern "C" int id11b_dev_refine_translations(const double* xyz, const double* omega,
                                             const int64_t* offsets, int32_t ngrains,
                                             const double* ubis, double* translations,
                                             double omegasign, double wvln, double wedge,
                                             double chi, double tol, int iters, double* cost,
                                             int32_t* npk, double* ubis_refit, void* stream) {
    if (ngrains < 0 || iters < 0 || iters > 1000 || !(tol > 0.) || !(wvln > 0.))
        return ID11B_ERR_ARG;
    if (ngrains == 0) return ID11B_OK;
    if (!xyz || !omega || !offsets || !ubis || !translations) return ID11B_ERR_ARG;
    Geo P;
    wedgechi(wedge, chi, P.m);
    P.omegasign = omegasign;
    P.ds = 1.0 / wvln;
    P.tol2 = tol * tol;
    // Shared memory for the CTAs that will be on an SM, the rest of its 228 KB as L1: each
    // pass reads the grain's peaks again (30 grains of 4,900 peaks, 196 KB each: 0.90 ms,
    // 1.15 with the split the driver takes).
    int dev = 0, sms = 0;
    ID11B_CHECK(cudaGetDevice(&dev));
    ID11B_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int each = (int)sizeof(double) * 3 * kKeep * kTT;
    const int ctas = std::min((ngrains - 1) / std::max(sms, 1) + 1, kResident);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[0].val.sharedMemCarveout = 100 * ctas * (each + 2048) / (228 * 1024) + 1;  // percent
    cfg.gridDim = dim3((unsigned)ngrains);
    cfg.blockDim = dim3(kTT);
    cfg.dynamicSmemBytes = each;
    cfg.stream = (cudaStream_t)stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    ID11B_CHECK(cudaLaunchKernelEx(&cfg, k_refine_translations, xyz, omega, offsets, ngrains, ubis,
                                   translations, P, iters, cost, npk, ubis_refit));
    return ID11B_OK;
}
