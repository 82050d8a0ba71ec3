// Batched per-grain refinement over CSR peak lists (score_and_refine x iters).
//
// Grain g owns the g-vectors gv[off[g] : off[g+1]] (20 .. 2000 peaks each in
// the uneven workload) and `iters` rounds of the reference's score_and_refine
// (ImageD11 src/closest.c:267-345) are applied to its UBI.  One CTA (128,
// 256 or 512 threads, chosen from the largest grain) refines one grain at a
// time and runs all rounds itself: per round, every thread tests its peaks
// with the reference's exact FP64 arithmetic and accumulates the accepted
// peaks' normal-equation terms, the CTA reduces them in a fixed tree (exchanges
// that leave one sum per lane, then the warps in order), and nine lanes of the
// first warp apply the reference's update (one cofactor / one UB element each;
// the same expressions as inverse3x3, so the result equals the single-thread
// update bit for bit).
//
// Persistent mode (queue != null): a grid sized to the GPU, each CTA's first
// grain its own index, the others from an atomic work counter read while the
// grain before is refined, in the caller's order -- largest grains first (LPT)
// keeps the tail short.  No CTA ever waits on another, so there is nothing to
// time out.  Plain mode (queue == null): CTA b refines grain order[b]; used
// one launch per round as the straightforward baseline.
//
// Peaks are evaluated in exact FP64 here: refinement segments are a grain's
// own peaks, nearly all accepted, and every accepted pair needs its FP64
// g-vector and exact drlv2 anyway, so an FP32 pre-screen would only add work.
#include "common.cuh"

namespace id11b {

struct RefineSmem {
    double m[27], ubi[9];
};

// Compensated FP32 accumulation (the F32C variant): a sum kept as s + c with
// every addition's rounding error recovered exactly (TwoSum) and every
// product's by an FMA (TwoProduct), Ogita, Rump and Oishi, "Accurate sum and
// dot product", SIAM J. Sci. Comput. 26 (2005) -- as accurate as a sum in
// twice the working precision.
__device__ __forceinline__ void comp_add(float& s, float& c, float x) {
    const float t = s + x;
    const float bp = t - s;
    c += (s - (t - bp)) + (x - bp);
    s = t;
}

// One round's pass over a thread's n peaks (every N-th of the grain's from first on),
// in the reference's FP64 arithmetic: the accepted peaks' normal-equation terms.  Two peaks a step,
// their tests side by side (each is a chain of dependent operations) and the
// next two's loads in flight; the segment is read-only and re-read every round,
// so later rounds hit L1.  The terms use fused multiply-adds: H (products of
// integers) is exact either way; each R term is rounded once instead of twice --
// R is order-dependent against the reference's sequential sum in any case.
__device__ __forceinline__ void add_peak(const double ih[3], const double g[3], double s,
                                         double acc[17], int& nacc) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) acc[3 * i + j] = fma(ih[j], g[i], acc[3 * i + j]);
    acc[9] = fma(ih[0], ih[0], acc[9]);
    acc[10] = fma(ih[1], ih[0], acc[10]);
    acc[11] = fma(ih[2], ih[0], acc[11]);
    acc[12] = fma(ih[1], ih[1], acc[12]);
    acc[13] = fma(ih[2], ih[1], acc[13]);
    acc[14] = fma(ih[2], ih[2], acc[14]);
    acc[15] = dadd(acc[15], s);
    nacc++;
}

template <int N>
__device__ __forceinline__ void refine_peaks(const double u[9], const double* __restrict__ first,
                                             int n, double tolsq, double acc[17], int& nacc) {
    double nxt[2][3];
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int i = 0; i < 3; i++)
            nxt[q][i] = q < n ? __ldg(first + 3 * q * N + i) : 0.;
    const double* p = first;
    for (int left = n; left > 0; left -= 2) {
        double g[2][3], ih[2][3];
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int i = 0; i < 3; i++) g[q][i] = nxt[q][i];
        p += 6 * N;
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (left > 2 + q)
#pragma unroll
                for (int i = 0; i < 3; i++) nxt[q][i] = __ldg(p + 3 * q * N + i);
        const double s0 = drlv2_exact(u, g[0][0], g[0][1], g[0][2], ih[0]);
        const double s1 = drlv2_exact(u, g[1][0], g[1][1], g[1][2], ih[1]);
        if (s0 < tolsq) add_peak(ih[0], g[0], s0, acc, nacc);
        if (left > 1 && s1 < tolsq) add_peak(ih[1], g[1], s1, acc, nacc);
    }
}

// The same in the F32C variant: FP32 screening with the proven band
// (score_batch.cu) for this UBI, compensated R and drlv2 sums, exact integer H.
template <int N>
__device__ __forceinline__ void refine_peaks_f32c(const double u[9],
                                                  const double* __restrict__ first, int n,
                                                  double tolsq, double gmax, double acc[17],
                                                  int& nacc) {
    float u32[9], rs[9], rc[9], ss32 = 0.f, sc32 = 0.f;
    int hint[6] = {0, 0, 0, 0, 0, 0};
    double S = 0.;
#pragma unroll
    for (int r = 0; r < 3; r++)
        S = fmax(S, fabs(u[3 * r]) + fabs(u[3 * r + 1]) + fabs(u[3 * r + 2]));
    const double E = 6.0 * 5.9604644775390625e-08 * S * (1. + 1e-15) * gmax;
    const double t = sqrt(tolsq);
    const double band = 1.25 * (3.0 * E * (2.0 * (t + 1e-3) + E) +
                                4.0 * 5.9604644775390625e-08 * (tolsq + 0.01));
    const float lo32 = __double2float_rd(tolsq - band), hi32 = __double2float_ru(tolsq + band);
#pragma unroll
    for (int e = 0; e < 9; e++) {
        u32[e] = __double2float_rn(u[e]);
        rs[e] = rc[e] = 0.f;
    }
    // kU peaks per lane per step: all their loads are issued before any is used
    constexpr int kU = 4;
    const double* p = first;
    for (int k = 0; k < n; k += kU, p += 3 * kU * N) {
        double gg[kU][3];
#pragma unroll
        for (int q = 0; q < kU; q++)
            if (k + q < n)
#pragma unroll
                for (int i = 0; i < 3; i++) gg[q][i] = __ldg(p + 3 * q * N + i);
#pragma unroll
        for (int q = 0; q < kU; q++) {
            if (k + q >= n) break;
            // g split exactly enough into hi + lo floats
            float gh[3], gl[3], ihf[3], d[3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                gh[i] = __double2float_rn(gg[q][i]);
                gl[i] = __double2float_rn(gg[q][i] - (double)gh[i]);
            }
            const float M = 12582912.0f;  // 1.5 * 2^23
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float h = fmaf(u32[3 * r + 2], gh[2],
                                     fmaf(u32[3 * r + 1], gh[1], u32[3 * r] * gh[0]));
                ihf[r] = __fsub_rn(__fadd_rn(h, M), M);
                d[r] = h - ihf[r];
            }
            float s32 = fmaf(d[2], d[2], fmaf(d[1], d[1], d[0] * d[0]));
            if (!(s32 < hi32)) continue;
            if (!(s32 < lo32)) {  // inside the band: the exact decision
                double ih[3];
                const double s = drlv2_exact(u, gg[q][0], gg[q][1], gg[q][2], ih);
                if (!(s < tolsq)) continue;
#pragma unroll
                for (int r = 0; r < 3; r++) ihf[r] = (float)ih[r];
                s32 = (float)s;
            }
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    // ih_j * g_i = ih_j * gh_i (TwoProduct) + ih_j * gl_i
                    const float pr = ihf[j] * gh[i];
                    const float pe = fmaf(ihf[j], gh[i], -pr);
                    comp_add(rs[3 * i + j], rc[3 * i + j], pr);
                    rc[3 * i + j] += pe + ihf[j] * gl[i];
                }
            const int a = (int)ihf[0], b = (int)ihf[1], c = (int)ihf[2];
            hint[0] += a * a;
            hint[1] += b * a;
            hint[2] += c * a;
            hint[3] += b * b;
            hint[4] += c * b;
            hint[5] += c * c;
            comp_add(ss32, sc32, s32);
            nacc++;
        }
    }
    // to FP64 for the fixed reduction: s + c, exact integers
#pragma unroll
    for (int e = 0; e < 9; e++) acc[e] = (double)rs[e] + (double)rc[e];
#pragma unroll
    for (int e = 0; e < 6; e++) acc[9 + e] = (double)hint[e];
    acc[15] = (double)ss32 + (double)sc32;
}

// `iters` rounds of one grain by N threads (tid of them; N == 32: one warp of the
// CTA by itself).  red: N / 32 rows of per-warp partial sums.  V > 1 (N == 32):
// the warp does the work of V warps in turn, peak by peak and sum by sum as they
// would, so the result has the same bits.
template <int N, bool F32C, int V = 1, class Len>
__device__ __forceinline__ void refine_grain(RefineSmem& sm, double (*red)[17], int tid, int g,
                                             double* __restrict__ ubis,
                                             const double* __restrict__ gv, int64_t k0, Len n,
                                             double tolsq, int iters, int* __restrict__ npk,
                                             double* __restrict__ mean, double gmax) {
    const int lane = tid & 31, w = tid >> 5;
    auto sync = [] {
        if (N == 32) __syncwarp(); else __syncthreads();
    };
    const int field = slot_of<17>(lane);
    if (tid < 9) sm.ubi[tid] = ubis[9 * (int64_t)g + tid];
    sync();
    // peaks of the thread that begins at `first`: an int whatever the grain's length
    auto count = [&](int first) { return (int)((n - first + (N * V - 1)) / (N * V)); };
    const int mine = count(tid);
    for (int it = 0; it < iters; it++) {
        double u[9];
#pragma unroll
        for (int e = 0; e < 9; e++) u[e] = sm.ubi[e];
        double part = 0.;
#pragma unroll 1
        for (int v = 0; v < V; v++) {
            const int first = tid + 32 * v;
            double acc[17];
#pragma unroll
            for (int f = 0; f < 17; f++) acc[f] = 0.;
            int nacc = 0;
            const int cnt = V == 1 ? mine : count(first);
            const double* p = gv + 3 * (k0 + first);
            if (F32C)
                refine_peaks_f32c<N * V>(u, p, cnt, tolsq, gmax, acc, nacc);
            else
                refine_peaks<N * V>(u, p, cnt, tolsq, acc, nacc);
            acc[16] = (double)nacc;
            part += ScatterSum<17, 16>::run(acc, lane);
        }
        if (field >= 0) red[w][field] = part;
        sync();
        if (w == 0) {
            double t = 0.;
            if (lane < 17)
                for (int q = 0; q < N / 32; q++) t += red[q][lane];
            // t: R in lanes 0 .. 8, H's upper triangle 9 .. 14, sum, n
            const double ss = __shfl_sync(0xffffffffu, t, 15);
            const long long np = (long long)__shfl_sync(0xffffffffu, t, 16);
            const double v = lsq_update_warp(t, lane < 9 ? sm.ubi[lane] : 0., sm.m, lane);
            if (lane < 9) sm.ubi[lane] = v;
            if (lane == 0 && it == iters - 1) {
                if (npk) npk[g] = (int)np;
                if (mean) mean[g] = np > 0 ? ddiv(ss, (double)np) : 0.;
            }
        }
        sync();
    }
    if (tid < 9) ubis[9 * (int64_t)g + tid] = sm.ubi[tid];
    sync();
}

// Persistent mode with more grains than CTAs: CTAs of NT threads take grains of
// more than `solo` peaks whole; from the first smaller one on, each of a CTA's
// warps takes grains by itself, so that the rounds' fixed part (the reduction
// and the 3x3 solves, which one warp does) of several grains overlap.  A larger
// grain met after that (an order that is not by size) is done by one warp as the
// CTA would.  So the order of a grain's sums, and with it the last bits of its UBI,
// follows from its size, from NT and, for grains of up to `solo` peaks, from how many
// more grains than CTAs the call has; never from the order of the grains or of the
// CTAs.  (One order for both, kept here, would cost more than it gives: the CTA's by
// one warp 2,000 grains of 20 .. 2,000 peaks 39 -> 49 us, one warp's where there are
// few grains 500 of 20 .. 768 peaks 16.4 -> 22.6 us.)
//
// Bound: instruction issue and FP64 latency at 16 resident warps (116 registers),
// then the largest grains' own five rounds.  2,000 grains of 20 ..
// 2,000 peaks (859k), five rounds: 36.6 us with 128 threads, 42 with 64; 55.9 (64)
// and 80.2 (128) with a CTA for every grain, 17 warp sums and five barriers a
// round.  500 such grains 36.0 -> 17.0, 8,000 of up to 400 peaks, three rounds, 86
// -> 35 us.
//
// Solo grains of up to 256, 512, 768 and 1,024 at 128 threads, five rounds, us (the
// launch among others): 1,000 grains of 20 .. 2,000 peaks 30.3, 30.6, 30.3, 30.6; 2,000 of up to
// 1,000 37.4, 33.4, 34.8, 37.1 and of up to 2,000 45.9, 45.0, 39.1, 43.2; 4,000 of up
// to 1,000 57.3, 53.0, 50.2, 54.0; 8,000 of up to 2,000 119, 110, 106, 109; 3,000 of
// 600 .. 760 75.2, 75.0, 78.1, 78.1 and of 780 .. 1,000 84.1, 84.0, 84.1, 94.1.  768
// is the best or within 4% of it on all of them.
// The F32C variant does more per peak, so fewer go to one warp where there are few
// grains per CTA, and more where there are many.  192, 384, 768, 1,024: 500 of up to
// 2,000 peaks 37.6, 38.0, 45.2, 48.7; 1,000 48.6, 53.2, 54.8, 55.4; 2,000 73.3, 69.8,
// 73.9, 75.4; 4,000 of up to 1,000 92.3, 86.7, 79.3, 83.1; 8,000 of up to 2,000 221,
// 207, 194, 192; 3,000 of 600 .. 760 135, 134, 106, 106 and of 780 .. 1,000 154, 153,
// 154, 133; 20,000 of 300 .. 500 644, 508, 371, 371.  With a CTA of 64 threads for
// every grain 2,000 of up to 2,000 took 86, the last three 124, 144, 551.
constexpr int kSoloFp64 = 768, kSoloF32c = 384, kSoloF32cMany = 1024;
constexpr int kManyPerCta = 6;

template <int NT, bool F32C = false>
__global__ void __launch_bounds__(NT)
k_refine_csr(double* __restrict__ ubis, const double* __restrict__ gv,
             const int64_t* __restrict__ off, const int* __restrict__ order, int ngrains,
             double tolsq, int iters, int* __restrict__ queue, int* __restrict__ npk,
             double* __restrict__ mean, double gmax) {
    __shared__ RefineSmem sm[NT / 32];
    __shared__ double s_red[NT / 32][17];
    __shared__ int s_next;
    const int solo = !F32C ? kSoloFp64 :
                     ngrains / kManyPerCta > (int)gridDim.x ? kSoloF32cMany : kSoloF32c;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int slot = blockIdx.x;
    while (slot < ngrains) {
        const int g = order ? order[slot] : slot;
        const int64_t k0 = off[g];
        const int64_t n = off[g + 1] - k0;
        if (NT > 32 && queue && ngrains > (int)gridDim.x && n <= solo) break;
        if (tid == 0) s_next = queue ? (int)gridDim.x + atomicAdd(queue, 1) : ngrains;
        refine_grain<NT, F32C>(sm[0], s_red, tid, g, ubis, gv, k0, n, tolsq, iters, npk, mean,
                               gmax);
        slot = s_next;
        if (NT == 32) __syncwarp(); else __syncthreads();
    }
    if (NT == 32) return;
    // one warp per grain: warp 0 begins with the CTA's
    int mine = slot;
    if (w > 0) {
        mine = ngrains;
        if (slot < ngrains) {
            if (lane == 0) mine = (int)gridDim.x + atomicAdd(queue, 1);
            mine = __shfl_sync(0xffffffffu, mine, 0);
        }
    }
    while (mine < ngrains) {
        const int g = order ? order[mine] : mine;
        const int64_t k0 = off[g];
        const int64_t n = off[g + 1] - k0;
        int next = 0;
        if (lane == 0) next = (int)gridDim.x + atomicAdd(queue, 1);
        if (n <= solo)
            refine_grain<32, F32C>(sm[w], s_red + w, lane, g, ubis, gv, k0, (int)n, tolsq, iters,
                                   npk, mean, gmax);
        else
            refine_grain<32, F32C, NT / 32>(sm[w], s_red + w, lane, g, ubis, gv, k0, n, tolsq,
                                            iters, npk, mean, gmax);
        mine = __shfl_sync(0xffffffffu, next, 0);
    }
}

static int sm_count_rc() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}

}  // namespace id11b

using namespace id11b;

template <int NT, bool F32C = false>
static int launch_refine(double* ubis, const double* gv, const int64_t* offsets,
                         const int32_t* order, int32_t ngrains, double tolsq, int iters,
                         int* queue, int32_t* npk, double* mean, cudaStream_t st,
                         double gmax = 0.) {
    int grid = ngrains;
    if (queue) {
        static int occ = 0;
        if (!occ) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_refine_csr<NT, F32C>, NT, 0);
            if (occ < 1) occ = 1;
        }
        const int cap = sm_count_rc() * occ;
        grid = ngrains < cap ? ngrains : cap;
    }
    k_refine_csr<NT, F32C><<<grid, NT, 0, st>>>(ubis, gv, offsets, order, ngrains, tolsq, iters,
                                                queue, npk, mean, gmax);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int64_t id11b_refine_csr_workspace_bytes(void) { return 256; }

extern "C" int id11b_dev_refine_csr(double* ubis, const double* gv, const int64_t* offsets,
                                    const int32_t* order, int32_t ngrains, double tol,
                                    int iters, int persistent, int threads, int32_t* npk,
                                    double* mean_drlv2, void* workspace, int64_t ws_bytes,
                                    void* stream) {
    if (ngrains < 0 || iters < 0) return ID11B_ERR_ARG;
    if (ngrains > 0 && (!ubis || !offsets)) return ID11B_ERR_ARG;
    if (persistent && (!workspace || ws_bytes < id11b_refine_csr_workspace_bytes()))
        return ID11B_ERR_ARG;
    if (threads != 0 && threads != 32 && threads != 64 && threads != 128 && threads != 256 &&
        threads != 512)
        return ID11B_ERR_ARG;
    if (ngrains == 0 || iters == 0) return ID11B_OK;
    cudaStream_t st = (cudaStream_t)stream;
    int* queue = nullptr;
    if (persistent) {
        queue = (int*)workspace;
        ID11B_CHECK(cudaMemsetAsync(queue, 0, sizeof(int), st));
    }
    const double tolsq = tol * tol;
    switch (threads) {
        case 32: return launch_refine<32>(ubis, gv, offsets, order, ngrains, tolsq, iters, queue, npk, mean_drlv2, st);
        case 64: return launch_refine<64>(ubis, gv, offsets, order, ngrains, tolsq, iters, queue, npk, mean_drlv2, st);
        case 256: return launch_refine<256>(ubis, gv, offsets, order, ngrains, tolsq, iters, queue, npk, mean_drlv2, st);
        case 512: return launch_refine<512>(ubis, gv, offsets, order, ngrains, tolsq, iters, queue, npk, mean_drlv2, st);
        default: return launch_refine<128>(ubis, gv, offsets, order, ngrains, tolsq, iters, queue, npk, mean_drlv2, st);
    }
}

// The same rounds with FP32 screening (the proven band, FP64 inside it) and
// compensated FP32 normal-equation sums (integer H), FP64 3x3 solves: the
// accumulation the batched design could use instead of FP64 sums.  gmax:
// bound on every |g_j| of the segments (the band's input); g-vectors beyond
// 1024 or non-finite are not supported by this variant (ID11B_ERR_ARG).
extern "C" int id11b_dev_refine_csr_f32c(double* ubis, const double* gv, const int64_t* offsets,
                                         const int32_t* order, int32_t ngrains, double tol,
                                         int iters, double gmax, int32_t* npk,
                                         double* mean_drlv2, void* workspace, int64_t ws_bytes,
                                         void* stream) {
    if (ngrains < 0 || iters < 0 || !(gmax >= 0.) || !(gmax <= 1024.) || !(tol >= 0.) ||
        !(tol < 0.4))
        return ID11B_ERR_ARG;
    if (ngrains > 0 && (!ubis || !offsets)) return ID11B_ERR_ARG;
    if (!workspace || ws_bytes < id11b_refine_csr_workspace_bytes()) return ID11B_ERR_ARG;
    if (ngrains == 0 || iters == 0) return ID11B_OK;
    cudaStream_t st = (cudaStream_t)stream;
    int* queue = (int*)workspace;
    ID11B_CHECK(cudaMemsetAsync(queue, 0, sizeof(int), st));
    return launch_refine<128, true>(ubis, gv, offsets, order, ngrains, tol * tol, iters, queue,
                                   npk, mean_drlv2, st, gmax);
}
