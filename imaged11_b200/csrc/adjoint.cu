// Residuals of assigned peaks, their hand-written adjoint, and the geometry
// map, all on the device (FP64).
//
// Geometry parameters (12, device memory, in this order): distance,
// y_center, z_center, tilt_x, tilt_y, tilt_z (radians), wavelength, wedge,
// chi (degrees), t_x, t_y, t_z.  Fixed detector constants (7, host): y_size,
// z_size, omegasign, o11, o12, o21, o22.  Every launch rebuilds
//   r = R3(tilt_x).R2(tilt_y).R1(tilt_z).flip   (ImageD11/transform.py:51-82, :688-692)
//   M = W(wedge).C(chi)                          (src/cdiffraction.c:117-142)
// from the device copy of the parameters, so a step of an optimiser never
// copies the geometry to the host.
//
// Forward model for peak k of grain G (peaks stored grain by grain, CSR):
//   detector -> lab (ImageD11 src/cdiffraction.c:190-224)
//     v1 = (f - y_center) * y_size,  v2 = (s - z_center) * z_size
//     xyz = r[:,1] v1 + r[:,2] v2 + (distance, 0, 0)
//   lab -> g (ImageD11 src/cdiffraction.c:112-168)
//     u = Omega(w)^T t,  o = M u,  d = xyz - o,  dh = d / |d|
//     k = (dh - x) / wavelength,  v = M^T k,  g = Omega(w) v
//   residual  res = UBI_G . g - h_k          (h_k: the peak's assigned hkl)
//
// Backward, given a_res = dL/d res for every peak (reverse mode, per peak):
//   dL/dUBI_G += a_res g^T             a_g = UBI_G^T a_res
//   a_v = Omega^T a_g                  a_k = M a_v,   dL/dM += k a_v^T
//   dL/dwavelength += -(a_k . k) / wavelength
//   a_dh = a_k / wavelength            a_d = (a_dh - dh (dh . a_dh)) / |d|
//   a_xyz = a_d                        a_o = -a_d,    dL/dM += a_o u^T
//   a_u = M^T a_o                      dL/dt += Omega a_u
//   dL/dr[:,1] += a_xyz v1,  dL/dr[:,2] += a_xyz v2,  sum a_xyz (-> distance, centres)
// and, once per launch, dL/dM and dL/dr are contracted with dM/d(wedge, chi)
// and dr/d(tilts), the centre and distance terms with r and the pixel sizes
// (k_finish).
//
// One CTA (one to four warps, by the number of grains) takes grains in a fixed
// stride, accumulates a grain's peaks in registers and reduces them in a fixed
// tree; the geometry's sums stay one per lane from grain to grain and go out as
// one row per CTA, and one CTA then sums the rows in order.  Every result is
// deterministic.
//
// Variable projection (MODE 3): each grain's UBI is first solved in closed
// form for the current g (UBI = (sum h g^T)(sum g g^T)^-1, the least-squares
// fit), then the loss and geometry gradient are taken at that UBI.  At the
// least-squares UBI dL/dUBI = 0, so the gradient of the projected loss with
// respect to the geometry equals the partial derivative computed here.
#include <algorithm>

#include "common.cuh"

namespace id11b {

constexpr int kAT = 64;         // threads per CTA of k_bragg
constexpr int kNP = 12;         // geometry parameters
constexpr int kGlob = 22;       // dM(9) -dlam*wavelength(1) dt(3) sum_axyz(3) dR1(3) dR2(3)
constexpr int kPart = kGlob + 1;  // + sum of squared residuals
constexpr int kRow = 32;        // doubles per CTA row of sums
constexpr int kMaxRows = 4096;  // CTAs of a launch that sums rows

struct AdjDet {
    double y_size, z_size, omegasign, o11, o12, o21, o22;
};

struct AdjGeom {
    double r[9];        // detector rotation . flip (row-major)
    double M[9];        // chi.wedge
    double t[3];        // grain-origin translation
    double wavelength, inv_wavelength, distance, y_center, z_center, y_size, z_size, omegasign;
};

struct PeakState {
    double so, co, u[3], v1, v2, dh[3], rn, k[3], g[3];  // rn = 1 / |d|
};

__device__ __forceinline__ void mat3mul(const double* a, const double* b, double* c) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            c[3 * i + j] = a[3 * i] * b[j] + a[3 * i + 1] * b[3 + j] + a[3 * i + 2] * b[6 + j];
}

// The rotation factors of r and M and their derivatives:
// R[0..2] = R3(tilt_x), R2(tilt_y), R1(tilt_z); dR the same differentiated;
// F the detector flip; W, C and dW, dC per radian.
struct RotFactors {
    double R[3][9], dR[3][9], F[9], W[9], C[9], dW[9], dC[9];
};

// sin and cos of the five angles, each taken by its own lane (a warp; the
// chain of five would be most of the kernels' start-up): sc = sin, cos of
// tilt_x, tilt_y, tilt_z, wedge, chi
__device__ __forceinline__ void angle_sincos(const double* __restrict__ p, double sc[10]) {
    const int lane = threadIdx.x & 31;
    const double rad = 3.14159265358979323846 / 180.0;
    double a = 0., s, c;
    if (lane < 3) a = p[3 + lane];
    if (lane == 3 || lane == 4) a = p[4 + lane] * rad;
    sincos(a, &s, &c);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        sc[2 * k] = __shfl_sync(0xffffffffu, s, k);
        sc[2 * k + 1] = __shfl_sync(0xffffffffu, c, k);
    }
}

__device__ void rot_factors(const double sc[10], const AdjDet& D, RotFactors& f) {
    const double sx = sc[0], cx = sc[1], sy = sc[2], cy = sc[3], sz = sc[4], cz = sc[5],
                 sw = sc[6], cw = sc[7], sk = sc[8], ck = sc[9];
    const double R3[9] = {1, 0, 0, 0, cx, -sx, 0, sx, cx};
    const double R2[9] = {cy, 0, sy, 0, 1, 0, -sy, 0, cy};
    const double R1[9] = {cz, -sz, 0, sz, cz, 0, 0, 0, 1};
    const double dR3[9] = {0, 0, 0, 0, -sx, -cx, 0, cx, -sx};
    const double dR2[9] = {-sy, 0, cy, 0, 0, 0, -cy, 0, -sy};
    const double dR1[9] = {-sz, -cz, 0, cz, -sz, 0, 0, 0, 0};
    const double F[9] = {1, 0, 0, 0, D.o22, D.o21, 0, D.o12, D.o11};
    const double W[9] = {cw, 0, -sw, 0, 1, 0, sw, 0, cw};
    const double C[9] = {1, 0, 0, 0, ck, -sk, 0, sk, ck};
    const double dW[9] = {-sw, 0, -cw, 0, 0, 0, cw, 0, -sw};
    const double dC[9] = {0, 0, 0, 0, -sk, -ck, 0, ck, -sk};
#pragma unroll
    for (int e = 0; e < 9; e++) {
        f.R[0][e] = R3[e];
        f.R[1][e] = R2[e];
        f.R[2][e] = R1[e];
        f.dR[0][e] = dR3[e];
        f.dR[1][e] = dR2[e];
        f.dR[2][e] = dR1[e];
        f.F[e] = F[e];
        f.W[e] = W[e];
        f.C[e] = C[e];
        f.dW[e] = dW[e];
        f.dC[e] = dC[e];
    }
}

// a.b.c.F with one of a, b, c replaced by its derivative (which = 0, 1, 2)
// or none (which = -1).
__device__ void rot_product(const RotFactors& f, int which, double out[9]) {
    double ab[9], abc[9];
    mat3mul(which == 0 ? f.dR[0] : f.R[0], which == 1 ? f.dR[1] : f.R[1], ab);
    mat3mul(ab, which == 2 ? f.dR[2] : f.R[2], abc);
    mat3mul(abc, f.F, out);
}

__device__ void make_geom(const double* p, const double sc[10], const AdjDet& D, AdjGeom& P) {
    RotFactors f;
    rot_factors(sc, D, f);
    rot_product(f, -1, P.r);
    mat3mul(f.W, f.C, P.M);
    P.t[0] = p[9];
    P.t[1] = p[10];
    P.t[2] = p[11];
    P.wavelength = isinf(p[6]) ? 0. : p[6];  // (div_by's remainder; the quotient is 0)
    P.inv_wavelength = 1.0 / p[6];
    P.distance = p[0];
    P.y_center = p[1];
    P.z_center = p[2];
    P.y_size = D.y_size;
    P.z_size = D.z_size;
    P.omegasign = D.omegasign;
}

// sin and cos of the peak's omega * omegasign: from the table made by
// id11b_dev_omega_sincos when one is given (omega is fixed for a peak, so
// an optimiser's evaluations need not repeat them), else computed here
__device__ __forceinline__ void peak_sincos(const AdjGeom& P, const double* __restrict__ omega,
                                            const double* __restrict__ osc, int64_t kk,
                                            double& so, double& co) {
    if (osc) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(osc) + kk);
        so = v.x;
        co = v.y;
    } else {
        sincos(3.14159265358979323846 / 180.0 * omega[kk] * P.omegasign, &so, &co);
    }
}

// a / y given ry = 1 / y rounded: the quotient's remainder corrects the product
// (Markstein's division; three operations, the rounding is that of a division but
// for rare last bits).  An infinite y is passed as 0: its remainder would be NaN.
__device__ __forceinline__ double div_by(double a, double y, double ry) {
    const double q = a * ry;
    return fma(fma(-q, y, a), ry, q);
}

__device__ __forceinline__ void forward_peak(const AdjGeom& P, double s, double f, double so,
                                             double co, PeakState& q) {
    q.so = so;
    q.co = co;
    q.v1 = (f - P.y_center) * P.y_size;
    q.v2 = (s - P.z_center) * P.z_size;
    double xyz[3];
#pragma unroll
    for (int j = 0; j < 3; j++) xyz[j] = P.r[3 * j + 1] * q.v1 + P.r[3 * j + 2] * q.v2;
    xyz[0] += P.distance;
    q.u[0] = q.co * P.t[0] - q.so * P.t[1];
    q.u[1] = q.so * P.t[0] + q.co * P.t[1];
    q.u[2] = P.t[2];
    double d[3];
#pragma unroll
    for (int i = 0; i < 3; i++)
        d[i] = xyz[i] - (P.M[3 * i] * q.u[0] + P.M[3 * i + 1] * q.u[1] + P.M[3 * i + 2] * q.u[2]);
    q.rn = rsqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
#pragma unroll
    for (int i = 0; i < 3; i++) q.dh[i] = d[i] * q.rn;
    // divided, not multiplied by a rounded 1/wavelength: the rounding then
    // stays independent from peak to peak as wavelength varies
    q.k[0] = div_by(q.dh[0] - 1.0, P.wavelength, P.inv_wavelength);
    q.k[1] = div_by(q.dh[1], P.wavelength, P.inv_wavelength);
    q.k[2] = div_by(q.dh[2], P.wavelength, P.inv_wavelength);
    double v[3];
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] = P.M[i] * q.k[0] + P.M[3 + i] * q.k[1] + P.M[6 + i] * q.k[2];
    q.g[0] = q.co * v[0] + q.so * v[1];
    q.g[1] = -q.so * v[0] + q.co * v[1];
    q.g[2] = v[2];
}

// Reverse-mode terms of one peak given a_res; gl = the 22 global sums.
__device__ __forceinline__ void adjoint_peak(const AdjGeom& P, const PeakState& q,
                                             const double U[9], const double ar[3],
                                             double* dU, double* gl) {
    if (dU) {
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) dU[3 * i + j] += ar[i] * q.g[j];
    }
    double ag[3], av[3], ak[3];
#pragma unroll
    for (int j = 0; j < 3; j++) ag[j] = U[j] * ar[0] + U[3 + j] * ar[1] + U[6 + j] * ar[2];
    av[0] = q.co * ag[0] - q.so * ag[1];
    av[1] = q.so * ag[0] + q.co * ag[1];
    av[2] = ag[2];
#pragma unroll
    for (int i = 0; i < 3; i++)
        ak[i] = P.M[3 * i] * av[0] + P.M[3 * i + 1] * av[1] + P.M[3 * i + 2] * av[2];
    // dL/dM from v = M^T k: dM[j][i] += k_j av_i
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
        for (int i = 0; i < 3; i++) gl[3 * j + i] += q.k[j] * av[i];
    // dL/dwavelength = -(sum of ak.k) / wavelength, divided once at the end
    gl[9] += ak[0] * q.k[0] + ak[1] * q.k[1] + ak[2] * q.k[2];
    const double dd = q.dh[0] * ak[0] + q.dh[1] * ak[1] + q.dh[2] * ak[2];
    const double rl = q.rn * P.inv_wavelength;
    double ad[3];
#pragma unroll
    for (int i = 0; i < 3; i++) ad[i] = (ak[i] - q.dh[i] * dd) * rl;
    // o = M u: dM[i][j] += a_o_i u_j with a_o = -a_d
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) gl[3 * i + j] -= ad[i] * q.u[j];
    double au[3];
#pragma unroll
    for (int j = 0; j < 3; j++) au[j] = -(P.M[j] * ad[0] + P.M[3 + j] * ad[1] + P.M[6 + j] * ad[2]);
    gl[10] += q.co * au[0] + q.so * au[1];
    gl[11] += -q.so * au[0] + q.co * au[1];
    gl[12] += au[2];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        gl[13 + i] += ad[i];
        gl[16 + i] += ad[i] * q.v1;
        gl[19 + i] += ad[i] * q.v2;
    }
}

// Fixed-order CTA reduction of acc[NA]: warp butterflies, then the warps'
// partials summed in warp order.  Result in red[0][e] for every thread.
template <int NA>
__device__ __forceinline__ void cta_reduce(double* acc, double (*red)[NA]) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
#pragma unroll
    for (int e = 0; e < NA; e++) acc[e] = warp_sum(acc[e]);
    if (lane == 0)
#pragma unroll
        for (int e = 0; e < NA; e++) red[w][e] = acc[e];
    __syncthreads();
    for (int e = tid; e < NA; e += kAT) {
        double t = red[0][e];
        for (int q = 1; q < kAT / 32; q++) t += red[q][e];
        red[0][e] = t;
    }
    __syncthreads();
}

// The grain's least-squares UBI from the sums A = sum h g^T (9) and
// B = sum g g^T (6, upper triangle): UBI = A B^-1, element `lane` of it, by one
// warp (each lane one cofactor and one division).  B is positive
// semi-definite; fewer than three independent g leave it singular up to
// rounding, so the test is relative: det <= 1e-10 trace^3 counts as singular
// (UBI 0).
// ab, B: shared memory (B: nine doubles of scratch).
__device__ __forceinline__ double best_ubi(const double* ab, double* B, int lane) {
    const int e = lane < 9 ? lane : 0, i = e / 3, j = e - 3 * i;
    const int lo = min(i, j), hi = max(i, j);
    if (lane < 9) B[e] = ab[9 + hi + lo + (lo > 0)];  // 00 01 02 11 12 22
    __syncwarp();
    const double tr = B[0] + B[4] + B[8];
    const double det = B[0] * (B[4] * B[8] - B[5] * B[7]) - B[1] * (B[3] * B[8] - B[5] * B[6]) +
                       B[2] * (B[3] * B[7] - B[4] * B[6]);
    const double dx = det3_exact(B);
    const bool ok = det > 1e-10 * tr * tr * tr && dx != 0.;
    const double bi = ok ? inv3_elem(B, dx, e) : 0.;
    double x = 0.;
#pragma unroll
    for (int k = 0; k < 3; k++)
        x += ab[3 * i + k] * __shfl_sync(0xffffffffu, bi, 3 * k + j);
    return x;
}

// What the kernels read of a peak (H: its hkl too)
struct PeakIn {
    double s, f, so, co, h[3];
};

template <bool H>
__device__ __forceinline__ void load_peak(const AdjGeom& P, const double* __restrict__ sc,
                                          const double* __restrict__ fc,
                                          const double* __restrict__ omega,
                                          const double* __restrict__ osc,
                                          const double* __restrict__ hkl, int64_t kk, PeakIn& x) {
    x.s = __ldg(sc + kk);
    x.f = __ldg(fc + kk);
    peak_sincos(P, omega, osc, kk, x.so, x.co);
    if (H)
#pragma unroll
        for (int i = 0; i < 3; i++) x.h[i] = __ldg(hkl + 3 * kk + i);
}

// MODE 0: residuals (+ g, + per-grain sum of squares); ubis == nullptr
//         gives g only.
// MODE 1: adjoint of given dL/dres.
// MODE 2: loss 0.5 sum res^2 and its gradient (a_res = res) in one pass.
// MODE 3: variable projection: least-squares UBI per grain, then MODE 2 at it.
// MODE 4: least-squares UBI per grain only.
//
// T threads per CTA, one grain at a time.  Bound: the FP64 pipe (80 operations a
// peak for a forward pass and its normal-equation sums, 170 with the reverse
// pass) at the 43 % of its rate that 10 or 12 resident warps reach (the sums and
// the peak's state are 168 registers); the next peak's loads are in flight while
// one is computed.  Projected loss of 20,000 grains, 7.8M peaks: 0.23 ms and 0.012
// for k_finish, from 0.52 and 0.12 ms with 64 threads a grain, full butterflies
// (19,000 shuffles a grain), one thread's 3x3 solve, a division for each of 1/|d|
// and /wavelength, and a row of sums per grain.  Gradient of 500 grains, 245k
// peaks: 15.2 + 6.3 -> 7.9 + 4.5 us.
template <int MODE>
__host__ __device__ constexpr int residual_warps() {
    // resident warps per SM compiled for: 12 (168 registers) for the projected
    // loss, 0.23 ms against 0.29 at 10; the gradient spills at 12 (500 grains: 9.4 us
    // against 7.9)
    return MODE == 3 ? 12 : MODE == 1 || MODE == 2 ? 8 : 16;
}

template <int MODE, int T>
__global__ void __launch_bounds__(T, residual_warps<MODE>() * 32 / T)
k_residual(const double* __restrict__ params, AdjDet D, const double* __restrict__ sc,
           const double* __restrict__ fc, const double* __restrict__ omega,
           const double* __restrict__ osc,
           const double* __restrict__ hkl, const int64_t* __restrict__ off,
           const double* __restrict__ ubis, int ngrains, double* __restrict__ res,
           double* __restrict__ gout, double* __restrict__ ssq,
           const double* __restrict__ ares, double* __restrict__ dubi,
           double* __restrict__ rows, double* __restrict__ ubis_out) {
    constexpr bool kAdj = MODE == 1 || MODE == 2 || MODE == 3;
    constexpr int kU = MODE == 1 || MODE == 2 ? 9 : 0;  // dL/dUBI beside the geometry's sums
    constexpr int W = T / 32;
    __shared__ AdjGeom sP;
    __shared__ double s_red[W][32];
    __shared__ double s_ab[15], s_B[9];
    __shared__ double s_U[9];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (w == 0) {
        double a[10];
        angle_sincos(params, a);
        if (lane == 0) make_geom(params, a, D, sP);
    }
    auto sync = [] {  // one warp needs no barrier of the CTA
        if (T == 32) __syncwarp(); else __syncthreads();
    };
    sync();
    const AdjGeom& P = sP;
    const int slot = slot_of<kU + kPart>(lane);
    double total = 0.;  // the lane's geometry sum, over the CTA's grains
    for (int G = blockIdx.x; G < ngrains; G += gridDim.x) {
        const int64_t k0 = off[G], k1 = off[G + 1];
        double U[9];
        if (MODE == 3 || MODE == 4) {
            double a[15];
#pragma unroll
            for (int e = 0; e < 15; e++) a[e] = 0.;
            PeakIn in;
            if (k0 + tid < k1) load_peak<true>(P, sc, fc, omega, osc, hkl, k0 + tid, in);
            for (int64_t kk = k0 + tid; kk < k1; kk += T) {
                const PeakIn x = in;  // the next peak's loads are in flight meanwhile
                if (kk + T < k1) load_peak<true>(P, sc, fc, omega, osc, hkl, kk + T, in);
                PeakState q;
                forward_peak(P, x.s, x.f, x.so, x.co, q);
                const double* h = x.h;
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) a[3 * i + j] += h[i] * q.g[j];
                a[9] += q.g[0] * q.g[0];
                a[10] += q.g[0] * q.g[1];
                a[11] += q.g[0] * q.g[2];
                a[12] += q.g[1] * q.g[1];
                a[13] += q.g[1] * q.g[2];
                a[14] += q.g[2] * q.g[2];
            }
            const int at = slot_of<15>(lane);
            const double v = ScatterSum<15, 16>::run(a, lane);
            if (at >= 0) s_red[w][at] = v;
            sync();
            if (w == 0) {
                if (lane < 15) {
                    double t = s_red[0][lane];
                    for (int q = 1; q < W; q++) t += s_red[q][lane];
                    s_ab[lane] = t;
                }
                __syncwarp();
                const double x = best_ubi(s_ab, s_B, lane);
                if (lane < 9) {
                    s_U[lane] = x;
                    if (ubis_out) ubis_out[9 * (int64_t)G + lane] = x;
                }
            }
            sync();
            if (MODE == 4) continue;
#pragma unroll
            for (int e = 0; e < 9; e++) U[e] = s_U[e];
        } else if (ubis) {
#pragma unroll
            for (int e = 0; e < 9; e++) U[e] = ubis[9 * (int64_t)G + e];
        } else {
#pragma unroll
            for (int e = 0; e < 9; e++) U[e] = 0.;
        }
        double acc[kU + kPart];
#pragma unroll
        for (int e = 0; e < kU + kPart; e++) acc[e] = 0.;
        PeakIn in;
        constexpr bool kH = MODE == 2 || MODE == 3;
        if (k0 + tid < k1) load_peak<kH>(P, sc, fc, omega, osc, hkl, k0 + tid, in);
        for (int64_t kk = k0 + tid; kk < k1; kk += T) {
            const PeakIn x = in;
            if (kk + T < k1) load_peak<kH>(P, sc, fc, omega, osc, hkl, kk + T, in);
            PeakState q;
            forward_peak(P, x.s, x.f, x.so, x.co, q);
            if (MODE == 0) {
                if (gout) {
#pragma unroll
                    for (int i = 0; i < 3; i++) gout[3 * kk + i] = q.g[i];
                }
                if (ubis) {
                    double ss = 0.;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const double ri = U[3 * i] * q.g[0] + U[3 * i + 1] * q.g[1] +
                                          U[3 * i + 2] * q.g[2] - hkl[3 * kk + i];
                        if (res) res[3 * kk + i] = ri;
                        ss += ri * ri;
                    }
                    acc[0] += ss;
                }
            } else if (kAdj) {
                double ar[3];
                if (MODE == 1) {
#pragma unroll
                    for (int i = 0; i < 3; i++) ar[i] = ares[3 * kk + i];
                } else {
#pragma unroll
                    for (int i = 0; i < 3; i++)
                        ar[i] = U[3 * i] * q.g[0] + U[3 * i + 1] * q.g[1] + U[3 * i + 2] * q.g[2] -
                                x.h[i];
                    acc[kU + kGlob] += ar[0] * ar[0] + ar[1] * ar[1] + ar[2] * ar[2];
                }
                adjoint_peak(P, q, U, ar, kU ? acc : nullptr, acc + kU);
            }
        }
        if (MODE == 0) {
            if (ssq) {
                const double v = warp_sum(acc[0]);
                if (lane == 0) s_red[w][0] = v;
                sync();
                if (tid == 0) {
                    double t = s_red[0][0];
                    for (int q = 1; q < W; q++) t += s_red[q][0];
                    ssq[G] = t;
                }
                sync();
            }
            continue;
        }
        const double v = ScatterSum<kU + kPart, 16>::run(acc, lane);
        if (slot >= kU) total += v;
        if (kU && dubi) {
            if (T == 32) {
                if (slot >= 0 && slot < kU) dubi[9 * (int64_t)G + slot] = v;
            } else {
                if (slot >= 0 && slot < kU) s_red[w][slot] = v;
                sync();
                if (tid < kU) {
                    double t = s_red[0][tid];
                    for (int q = 1; q < W; q++) t += s_red[q][tid];
                    dubi[9 * (int64_t)G + tid] = t;
                }
                sync();
            }
        }
    }
    if (!kAdj) return;
    if (slot >= kU) s_red[w][slot - kU] = total;
    sync();
    if (tid < kPart) {
        double t = s_red[0][tid];
        for (int q = 1; q < W; q++) t += s_red[q][tid];
        rows[(int64_t)blockIdx.x * kRow + tid] = t;
    }
}

// Sums the CTAs' rows in order (warp w takes rows w, w + 32, ..., a lane per
// column; then the warps in order) and maps the sums onto the 12 geometry
// parameters; loss = 0.5 * sum of squares.
__global__ void __launch_bounds__(1024)
k_finish(const double* __restrict__ rows, int nrows, const double* __restrict__ params,
         AdjDet D, double* __restrict__ grad, double* __restrict__ loss) {
    __shared__ double s_w[32][kRow + 1];
    __shared__ double col[kRow];
    __shared__ double s_dr[4][9], s_dm[2][9];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double t = 0.;
    if (lane < kPart) {
#pragma unroll 14
        for (int r = w; r < nrows; r += 32) t += rows[(int64_t)r * kRow + lane];
    }
    s_w[w][lane] = t;
    if (w == 0) {  // r and its derivatives by the tilts, M's by wedge and chi
        double a[10];
        angle_sincos(params, a);
        if (lane < 4) {
            RotFactors f;
            rot_factors(a, D, f);
            rot_product(f, lane - 1, s_dr[lane]);
            if (lane < 2) mat3mul(lane == 0 ? f.dW : f.W, lane == 0 ? f.C : f.dC, s_dm[lane]);
        }
    }
    __syncthreads();
    if (w < kPart) {  // warp w: column w over the 32 warps
        const double v = warp_sum(s_w[lane][w]);
        if (lane == 0) col[w] = v;
    }
    __syncthreads();
    const int e = threadIdx.x;
    if (e == 31 && loss) *loss = 0.5 * col[kGlob];
    if (!grad || e >= kNP) return;
    const double* dM = col;          // dL/dM (row-major)
    const double* A = col + 13;      // sum of dL/dxyz
    const double* dR1 = col + 16;    // dL/dr[:,1]
    const double* dR2 = col + 19;    // dL/dr[:,2]
    const double* r = s_dr[0];
    double g;
    if (e == 0) {
        g = A[0];
    } else if (e <= 2) {
        g = -(e == 1 ? D.y_size : D.z_size) * (r[e] * A[0] + r[3 + e] * A[1] + r[6 + e] * A[2]);
    } else if (e <= 5) {             // tilt_x, tilt_y, tilt_z
        const double* dr = s_dr[e - 2];
        g = 0.;
        for (int i = 0; i < 3; i++) g += dr[3 * i + 1] * dR1[i] + dr[3 * i + 2] * dR2[i];
    } else if (e == 6) {
        g = -col[9] / params[6];
    } else if (e <= 8) {
        const double* dm = s_dm[e - 7];
        g = 0.;
        for (int i = 0; i < 9; i++) g += dM[i] * dm[i];
        g *= 3.14159265358979323846 / 180.0;
    } else {
        g = col[e + 1];
    }
    grad[e] = g;
}

// Bragg angle of each assigned reflection computed from its grain's UB and
// its derivative, as ImageD11 src/deriv.c:38-53 (g_to_k) computes them:
//   g = UB h,  t = wavelength |g| / 2,  theta = asin(t) (degrees),
//   dtheta/dUB_ij = (180/pi) wavelength / (2 |g| sqrt(1 - t^2)) g_i h_j.
// BACKWARD: grad_ub_G = sum over the grain's peaks of a_theta dtheta/dUB,
// reduced in a fixed order.
template <bool BACKWARD>
__global__ void __launch_bounds__(kAT)
k_bragg(const double* __restrict__ ubs, const double* __restrict__ hkl,
        const int64_t* __restrict__ off, int ngrains, double wavelength,
        double* __restrict__ theta, double* __restrict__ jac,
        const double* __restrict__ atheta, double* __restrict__ gub) {
    __shared__ double s_red[kAT / 32][9];
    const double deg = 180.0 / 3.14159265358979323846;
    for (int G = blockIdx.x; G < ngrains; G += gridDim.x) {
        double B[9];
#pragma unroll
        for (int e = 0; e < 9; e++) B[e] = ubs[9 * (int64_t)G + e];
        double acc[9];
#pragma unroll
        for (int e = 0; e < 9; e++) acc[e] = 0.;
        for (int64_t kk = off[G] + threadIdx.x; kk < off[G + 1]; kk += kAT) {
            const double h[3] = {hkl[3 * kk], hkl[3 * kk + 1], hkl[3 * kk + 2]};
            double g[3];
#pragma unroll
            for (int i = 0; i < 3; i++) g[i] = B[3 * i] * h[0] + B[3 * i + 1] * h[1] + B[3 * i + 2] * h[2];
            const double modg = sqrt(g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
            const double t = wavelength * modg / 2.0;
            const double c = deg * wavelength / (2.0 * modg * sqrt(1.0 - t * t));
            if (BACKWARD) {
                const double a = atheta[kk] * c;
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) acc[3 * i + j] += a * g[i] * h[j];
            } else {
                theta[kk] = deg * asin(t);
                if (jac)
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) jac[9 * kk + 3 * i + j] = c * g[i] * h[j];
            }
        }
        if (BACKWARD) {
            cta_reduce<9>(acc, s_red);
            if (threadIdx.x < 9) gub[9 * (int64_t)G + threadIdx.x] = s_red[0][threadIdx.x];
            __syncthreads();
        }
    }
}

// sin and cos of omega * omegasign (degrees) per peak, interleaved
__global__ void k_omega_sincos(const double* __restrict__ omega, int64_t n, double omegasign,
                               double* __restrict__ out) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        double so, co;
        sincos(3.14159265358979323846 / 180.0 * omega[k] * omegasign, &so, &co);
        out[2 * k] = so;
        out[2 * k + 1] = co;
    }
}

static int adj_grid(int ngrains) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
    const int cap = sms * 16;
    return ngrains < cap ? ngrains : cap;
}

template <int MODE, int T>
static int residual_slots() {  // resident CTAs of k_residual<MODE, T> on the GPU
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_residual<MODE, T>, T, 0) !=
            cudaSuccess || per < 1)
        per = 1;
    return (sms > 0 ? sms : 148) * per;
}

// k_residual's launch: the widest CTA for which every grain has one of its own
// resident, so that few grains still fill the GPU (100 grains' gradient: 5.0 us
// with 128 threads, 6.3 with 64, 9.6 with 32), one warp each where there are more
// grains than that (20,000 projected: 0.23 ms with 32, 0.25 with 64, 0.30 with 128).
template <int MODE, class... A>
static int launch_residual(int ngrains, int* rows, cudaStream_t st, A... args) {
    // best_ubis takes the projected loss's width, and so gives its UBIs bit for bit
    constexpr int kAs = MODE == 4 ? 3 : MODE;
    static const int wide = residual_slots<kAs, 128>(), half = residual_slots<kAs, 64>(),
                     slots32 = residual_slots<MODE, 32>();
    int grid;
    if (ngrains <= wide) {
        grid = std::min(ngrains, kMaxRows);
        k_residual<MODE, 128><<<grid, 128, 0, st>>>(args...);
    } else if (ngrains <= half) {
        grid = std::min(ngrains, kMaxRows);
        k_residual<MODE, 64><<<grid, 64, 0, st>>>(args...);
    } else {
        grid = std::min(ngrains, std::min(slots32, kMaxRows));
        k_residual<MODE, 32><<<grid, 32, 0, st>>>(args...);
    }
    ID11B_CHECK_LAUNCH();
    if (rows) *rows = grid;
    return ID11B_OK;
}

static int adj_det(const double* d, AdjDet& D) {
    if (!d) return ID11B_ERR_ARG;
    D.y_size = d[0];
    D.z_size = d[1];
    D.omegasign = d[2];
    D.o11 = d[3];
    D.o12 = d[4];
    D.o21 = d[5];
    D.o22 = d[6];
    return ID11B_OK;
}

}  // namespace id11b

using namespace id11b;

extern "C" int64_t id11b_adjoint_workspace_bytes(int32_t ngrains) {
    return (int64_t)sizeof(double) * kRow *
           (ngrains > 0 ? (ngrains < kMaxRows ? ngrains : kMaxRows) : 1);
}

// omega_sincos (optional, 16-byte aligned): the table id11b_dev_omega_sincos
// makes for these peaks; NULL computes sin and cos of omega in the kernels
static bool osc_misaligned(const double* osc) { return osc && ((uintptr_t)osc & 15); }

extern "C" int id11b_dev_residuals(const double* params, const double* detector,
                                   const double* sc, const double* fc, const double* omega,
                                   const double* omega_sincos, const double* hkl,
                                   const int64_t* offsets, const double* ubis, int32_t ngrains,
                                   double* res, double* gvec, double* ssq, void* stream) {
    AdjDet D;
    if (!params || adj_det(detector, D) || ngrains < 0) return ID11B_ERR_ARG;
    if (osc_misaligned(omega_sincos)) return ID11B_ERR_ALIGN;
    if (ngrains == 0) return ID11B_OK;
    if (!offsets || !sc || !fc || !omega) return ID11B_ERR_ARG;
    if (ubis && (!hkl || !res)) return ID11B_ERR_ARG;
    if (!ubis && !gvec) return ID11B_ERR_ARG;
    double* const none = nullptr;
    return launch_residual<0>(ngrains, nullptr, (cudaStream_t)stream, params, D, sc, fc, omega,
                              omega_sincos, hkl, offsets, ubis, ngrains, res, gvec,
                              ubis ? ssq : none, (const double*)none, none, none, none);
}

extern "C" int id11b_dev_residuals_adjoint(const double* params, const double* detector,
                                           const double* sc, const double* fc,
                                           const double* omega, const double* omega_sincos,
                                           const double* hkl, const int64_t* offsets,
                                           const double* ubis, int32_t ngrains,
                                           const double* grad_res, double* grad_ubis,
                                           double* grad_params, void* workspace,
                                           int64_t ws_bytes, void* stream) {
    AdjDet D;
    if (!params || adj_det(detector, D) || ngrains < 0 || !grad_params) return ID11B_ERR_ARG;
    if (osc_misaligned(omega_sincos)) return ID11B_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    if (ngrains == 0) {
        ID11B_CHECK(cudaMemsetAsync(grad_params, 0, sizeof(double) * kNP, st));
        return ID11B_OK;
    }
    if (!offsets || !sc || !fc || !omega || !hkl || !ubis || !grad_res || !workspace)
        return ID11B_ERR_ARG;
    if (ws_bytes < id11b_adjoint_workspace_bytes(ngrains)) return ID11B_ERR_SIZE;
    double* rows = (double*)workspace;
    double* const none = nullptr;
    int nrows = 0;
    const int rc = launch_residual<1>(ngrains, &nrows, st, params, D, sc, fc, omega, omega_sincos,
                                      hkl, offsets, ubis, ngrains, none, none, none, grad_res,
                                      grad_ubis, rows, none);
    if (rc) return rc;
    k_finish<<<1, 1024, 0, st>>>(rows, nrows, params, D, grad_params, nullptr);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_residual_loss(const double* params, const double* detector,
                                       const double* sc, const double* fc, const double* omega,
                                       const double* omega_sincos, const double* hkl,
                                       const int64_t* offsets, const double* ubis,
                                       int32_t ngrains, double* loss, double* grad_ubis,
                                       double* grad_params, double* ubis_out, void* workspace,
                                       int64_t ws_bytes, void* stream) {
    AdjDet D;
    if (!params || adj_det(detector, D) || ngrains < 0 || !loss) return ID11B_ERR_ARG;
    if (!ubis && grad_ubis) return ID11B_ERR_ARG;
    if (osc_misaligned(omega_sincos)) return ID11B_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    if (ngrains == 0) {
        ID11B_CHECK(cudaMemsetAsync(loss, 0, sizeof(double), st));
        if (grad_params) ID11B_CHECK(cudaMemsetAsync(grad_params, 0, sizeof(double) * kNP, st));
        return ID11B_OK;
    }
    if (!offsets || !sc || !fc || !omega || !hkl || !workspace) return ID11B_ERR_ARG;
    if (ws_bytes < id11b_adjoint_workspace_bytes(ngrains)) return ID11B_ERR_SIZE;
    double* rows = (double*)workspace;
    double* const none = nullptr;
    int nrows = 0;
    const int rc =
        ubis ? launch_residual<2>(ngrains, &nrows, st, params, D, sc, fc, omega, omega_sincos, hkl,
                                  offsets, ubis, ngrains, none, none, none, (const double*)none,
                                  grad_ubis, rows, none)
             : launch_residual<3>(ngrains, &nrows, st, params, D, sc, fc, omega, omega_sincos, hkl,
                                  offsets, (const double*)none, ngrains, none, none, none,
                                  (const double*)none, none, rows, ubis_out);
    if (rc) return rc;
    k_finish<<<1, 1024, 0, st>>>(rows, nrows, params, D, grad_params, loss);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_best_ubis(const double* params, const double* detector,
                                   const double* sc, const double* fc, const double* omega,
                                   const double* omega_sincos, const double* hkl,
                                   const int64_t* offsets, int32_t ngrains, double* ubis_out,
                                   void* stream) {
    AdjDet D;
    if (!params || adj_det(detector, D) || ngrains < 0) return ID11B_ERR_ARG;
    if (osc_misaligned(omega_sincos)) return ID11B_ERR_ALIGN;
    if (ngrains == 0) return ID11B_OK;
    if (!offsets || !sc || !fc || !omega || !hkl || !ubis_out) return ID11B_ERR_ARG;
    double* const none = nullptr;
    return launch_residual<4>(ngrains, nullptr, (cudaStream_t)stream, params, D, sc, fc, omega,
                              omega_sincos, hkl, offsets, (const double*)none, ngrains, none, none,
                              none, (const double*)none, none, none, ubis_out);
}

extern "C" int id11b_dev_bragg_theta(const double* ubs, const double* hkl,
                                     const int64_t* offsets, int32_t ngrains, double wavelength,
                                     double* theta, double* dtheta_dub, void* stream) {
    if (ngrains < 0) return ID11B_ERR_ARG;
    if (ngrains == 0) return ID11B_OK;
    if (!ubs || !hkl || !offsets || !theta) return ID11B_ERR_ARG;
    k_bragg<false><<<adj_grid(ngrains), kAT, 0, (cudaStream_t)stream>>>(
        ubs, hkl, offsets, ngrains, wavelength, theta, dtheta_dub, nullptr, nullptr);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_bragg_theta_adjoint(const double* ubs, const double* hkl,
                                             const int64_t* offsets, int32_t ngrains,
                                             double wavelength, const double* grad_theta,
                                             double* grad_ubs, void* stream) {
    if (ngrains < 0) return ID11B_ERR_ARG;
    if (ngrains == 0) return ID11B_OK;
    if (!ubs || !hkl || !offsets || !grad_theta || !grad_ubs) return ID11B_ERR_ARG;
    k_bragg<true><<<adj_grid(ngrains), kAT, 0, (cudaStream_t)stream>>>(
        ubs, hkl, offsets, ngrains, wavelength, nullptr, nullptr, grad_theta, grad_ubs);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_omega_sincos(const double* omega, int64_t n, double omegasign,
                                      double* sincos_out, void* stream) {
    if (n < 0) return ID11B_ERR_ARG;
    if (n == 0) return ID11B_OK;
    if (!omega || !sincos_out) return ID11B_ERR_ARG;
    if ((uintptr_t)sincos_out & 15) return ID11B_ERR_ALIGN;
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, 148 * 32);
    k_omega_sincos<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(omega, n, omegasign,
                                                                      sincos_out);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}
