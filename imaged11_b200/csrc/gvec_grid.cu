// Reciprocal-space cell index over the g-vectors, and scoring by hkl lookup.
//
// The reference's score() (ImageD11 src/closest.c:227-248) tests every g
// against a UBI.  A g-vector is counted iff |UBI.g - round(UBI.g)|^2 < tol^2,
// i.e. iff it lies inside the ellipsoid of radius tol (in hkl units) around
// UB.hkl for hkl = round(UBI.g), UB = UBI^-1.  This file bins the g-vectors
// into a uniform grid of cells (square in y and z, x cut finer; x fastest, so
// a row of cells along x is one contiguous range of the cell-sorted g), then
// for each UBI enumerates
// the integer hkl whose ellipsoid can reach the data and tests only the g in
// the cells overlapping a conservative bounding box of that ellipsoid.  Every
// tested pair is evaluated with the reference's exact FP64 arithmetic
// (drlv2_exact) and counted only under its own hkl (ih == hkl), so each g is
// counted at most once and exactly when the reference counts it.
//
// Conservativeness: with d = UBI.g - hkl, g = UB.hkl + UB.d, so
// |g_j - (UB.hkl)_j| <= |d| * ||row j of UB||.  The box half-widths use
// (tol + 1e-6) in place of |d|: 1e-6 in hkl units is far above the FP64
// rounding of h, of UB = inv(UBI) (condition number capped at 1e6) and of
// UB.hkl (|hkl| capped).  Cell coordinates come from one monotone function
// of a coordinate, used by the build and the query alike, so a g inside the
// box is always inside the scanned cells.  UBIs outside the caps (non-finite,
// singular, ill-conditioned, or with more candidate hkl than g-vectors) are
// scored by a plain scan of every regular g; g-vectors outside the regular
// range (non-finite or |g_j| > 1024), or outside the cube and ball of radius
// rmax the index was built for, by a scan over that list.
#include <algorithm>

#include "grid.cuh"

namespace id11b {
namespace grid {

// scoring CTAs: warps (one per work item) and the resident CTAs per SM the
// register budget is compiled for.  Occupancy decides the speed of the
// latency-bound lookups: 20,000 grains assigned over 10M g took 9.5 ms at 1 x 24
// (80 registers) and 8.7 ms at 1 x 32 (64 registers, a few spilled).
#ifndef ID11B_GRID_WARPS
#define ID11B_GRID_WARPS 1
#endif
#ifndef ID11B_GRID_MINB
#define ID11B_GRID_MINB 32
#endif
constexpr int kSW = ID11B_GRID_WARPS;
constexpr int kST = 32 * kSW;

// ------------------------------------------------------------------ build --
// max |g_j| and max |g| over regular g, as float bits rounded up
__global__ void __launch_bounds__(kGT)
k_bounds(const double* __restrict__ gv, int64_t n, unsigned int* __restrict__ out) {
    float gm = 0.f, rm = 0.f;
    for (int64_t k = (int64_t)blockIdx.x * kGT + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * kGT) {
        double a = gv[3 * k], b = gv[3 * k + 1], c = gv[3 * k + 2];
        if (!regular(a, b, c)) continue;
        gm = fmaxf(gm, __double2float_ru(fmax(fabs(a), fmax(fabs(b), fabs(c)))));
        rm = fmaxf(rm, __double2float_ru(sqrt(a * a + b * b + c * c) * (1. + 1e-12)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
        rm = fmaxf(rm, __shfl_xor_sync(0xffffffffu, rm, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, __float_as_uint(gm));
        atomicMax(out + 1, __float_as_uint(rm));
    }
}

// Each g's cell counted, and its place among the cell's g in the order the
// atomics ran; flag: 1 for a g that no cell holds.  Writes the header.
__global__ void __launch_bounds__(kGT)
k_count(const double* __restrict__ gv, int64_t n, const Header H, Header* __restrict__ Hp,
        int* __restrict__ cnt, int* __restrict__ flag, int* __restrict__ place) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *Hp = H;
        flag[n] = 0;
    }
    for (int64_t k = (int64_t)blockIdx.x * kGT + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * kGT) {
        double a = gv[3 * k], b = gv[3 * k + 1], c = gv[3 * k + 2];
        const bool reg = indexed(a, b, c, H);
        flag[k] = reg ? 0 : 1;
        if (reg) place[k] = atomicAdd(cnt + cell_of(a, b, c, H), 1);
    }
}

// Exclusive scans of two arrays x[0 .. len) into y (16-byte aligned), the
// CTAs' totals in tot: blocks 0 .. nb - 1 of the first, then the second's.
struct ScanJob {
    const int* x;
    int64_t len;
    int* y;
    int* tot;
    int nb;
};

__device__ __forceinline__ void scan_load(const int* __restrict__ x, int64_t base, int64_t len,
                                          int v[4]) {
    if (base + 3 < len) {
        const int4 q = *reinterpret_cast<const int4*>(x + base);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = base + q < len ? x[base + q] : 0;
    }
}

__device__ __forceinline__ void scan_store(int* __restrict__ y, int64_t base, int64_t len,
                                           const int v[4]) {
    if (base + 3 < len) {
        *reinterpret_cast<int4*>(y + base) = make_int4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (base + q < len) y[base + q] = v[q];
    }
}

// pass 1: each CTA's kScanPer entries, from zero
__global__ void __launch_bounds__(kScanT) k_scan_local(ScanJob first, ScanJob second) {
    __shared__ int s_w[kScanT / 32];
    const bool two = (int)blockIdx.x >= first.nb;
    const ScanJob J = two ? second : first;
    const int blk = (int)blockIdx.x - (two ? first.nb : 0);
    const int64_t base = (int64_t)blk * kScanPer + 4 * threadIdx.x;
    int v[4];
    scan_load(J.x, base, J.len, v);
    const int sum = v[0] + v[1] + v[2] + v[3];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int total;
    const int excl = warp_excl_scan(sum, lane, total);
    if (lane == 31) s_w[wid] = total;
    __syncthreads();
    if (wid == 0) {
        int all;
        const int we = warp_excl_scan(s_w[lane], lane, all);
        s_w[lane] = we;  // exclusive over warps
        if (lane == 31) J.tot[blk] = all;
    }
    __syncthreads();
    int run = s_w[wid] + excl, out[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        out[q] = run;
        run += v[q];
    }
    scan_store(J.y, base, J.len, out);
}

// pass 2: the totals in place (one CTA per array, sequential chunks)
__global__ void __launch_bounds__(kScanT) k_scan_totals(ScanJob first, ScanJob second) {
    __shared__ int s_w[kScanT / 32];
    __shared__ int s_carry;
    const ScanJob J = blockIdx.x ? second : first;
    int* __restrict__ tot = J.tot;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int b0 = 0; b0 < J.nb; b0 += kScanT) {
        const int i = b0 + threadIdx.x;
        const int v = i < J.nb ? tot[i] : 0;
        int total;
        const int excl = warp_excl_scan(v, lane, total);
        if (lane == 31) s_w[wid] = total;
        __syncthreads();
        if (wid == 0) {
            int all;
            const int we = warp_excl_scan(s_w[lane], lane, all);
            s_w[lane] = we;
        }
        __syncthreads();
        const int carry = s_carry;
        if (i < J.nb) tot[i] = carry + s_w[wid] + excl;
        __syncthreads();
        if (threadIdx.x == kScanT - 1) s_carry = carry + s_w[wid] + excl + v;
        __syncthreads();
    }
}

// pass 3
__global__ void __launch_bounds__(kScanT) k_scan_add(ScanJob first, ScanJob second) {
    const bool two = (int)blockIdx.x >= first.nb;
    const ScanJob J = two ? second : first;
    const int blk = (int)blockIdx.x - (two ? first.nb : 0);
    const int64_t base = (int64_t)blk * kScanPer + 4 * threadIdx.x;
    const int add = J.tot[blk];
    int v[4];
    scan_load(J.y, base, J.len, v);
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] += add;
    scan_store(J.y, base, J.len, v);
}

// The g of each cell listed where the cell begins, in the order of their places;
// the g that no cell holds in their own list, by index.
__global__ void __launch_bounds__(kGT)
k_list_cells(const double* __restrict__ gv, int64_t n, const Header* __restrict__ Hp,
             const int* __restrict__ start, const int* __restrict__ place,
             int* __restrict__ list, const int* __restrict__ spos, int* __restrict__ spec) {
    const Header H = *Hp;
    for (int64_t k = (int64_t)blockIdx.x * kGT + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * kGT) {
        double a = gv[3 * k], b = gv[3 * k + 1], c = gv[3 * k + 2];
        if (!indexed(a, b, c, H))
            spec[spos[k]] = (int)k;
        else
            list[start[cell_of(a, b, c, H)] + place[k]] = (int)k;
    }
}

// Each listed g to its sorted position: within a cell by index (the layout, and so
// every result, does not depend on the order the atomics ran in) -- its rank among
// the cell's list, mostly of one to three -- with its FP64 coordinates, its index,
// and the FP32 (round to nearest) copy for screening and staging, the x cell (as
// int bits) in w.  One thread per place of the list: neighbours are in the same or
// the next cells, so everything but the read of the g itself is coalesced.
//
// Bound: the random 24-byte reads, and the counts' passes over the cells.  The
// build of 61k g (512k cells), 1.1M (8.1M) and 10.2M (10.2M): 32, 101 and 687 us;
// scattering every g by atomics and sorting each cell by one thread took 68, 232 and
// 4,173 us, and 20.6 ms where cells hold a hundred g and more (now 0.08).
__global__ void __launch_bounds__(kGT)
k_place(const double* __restrict__ gv, const Header* __restrict__ Hp,
        const int* __restrict__ start, const int* __restrict__ list, double* __restrict__ gs,
        int* __restrict__ gidx, float4* __restrict__ g4) {
    const Header H = *Hp;
    const int64_t nreg = start[H.ncells];
    for (int64_t at = (int64_t)blockIdx.x * kGT + threadIdx.x; at < nreg;
         at += (int64_t)gridDim.x * kGT) {
        const int k = list[at];
        const double a = gv[3 * (int64_t)k], b = gv[3 * (int64_t)k + 1],
                     c = gv[3 * (int64_t)k + 2];
        const int64_t cid = cell_of(a, b, c, H);
        const int p0 = start[cid], p1 = start[cid + 1];
        int p = p0;
        if (p1 - p0 > 1)
            for (int q = p0; q < p1; q++) p += list[q] < k;
        gs[3 * (int64_t)p] = a;
        gs[3 * (int64_t)p + 1] = b;
        gs[3 * (int64_t)p + 2] = c;
        gidx[p] = k;
        g4[p] = make_float4(__double2float_rn(a), __double2float_rn(b), __double2float_rn(c),
                            __int_as_float(coord_x(a, H)));
    }
}

// Per-warp queue of hkl that reach the data.  Enumeration: 32 (h, k) columns
// at a time, each lane solving for the range of l whose lattice point lies
// within rmax + |w| of the origin (every hkl whose box can reach a regular g
// is inside it), the 32 ranges flattened across the warp; candidates passing
// the box test are queued (packed hkl) in ballot order, and whenever 32 are
// queued the warp runs the 32 lookups together (lookup_batch).  The UBI's plan
// lives in shared memory, not in registers.
constexpr int kQueue = 64;
constexpr int kSeg = 160;    // row segments a warp lists before it scans their g
constexpr int kMark = 1024;  // g they may start within (one mark bit each)
// (2 and 2: 20,000 grains assigned over 10M g in 8.7 ms; 4 and 4, which spill more
// registers, 13.1 ms; 3 and 2 9.7 ms; 2 and 3 8.6 ms but refinement 1.35 -> 1.44 ms)
constexpr int kRowsAhead = 2;  // rows of cells whose bounds a lane loads together
constexpr int kGAhead = 2;     // steps of 32 g whose loads are in flight together

// Per-warp scratch of the lookups.
struct Batch {
    float4 c[32];                 // centres of the boxes being looked up
    unsigned long long hkl[32];
    int2 seg[kSeg];               // rows of cells with g: (first position - prefix, box)
    unsigned mark[kMark / 32];    // a bit at each segment's prefix
    float u[9];                   // the UBI in FP32
    // g that passed the screen, waiting for the FP64 evaluation (32 at a time)
    unsigned long long ch[32 * (kGAhead + 1)];
    int cp[32 * (kGAhead + 1)];
    float cs[32 * (kGAhead + 1)];  // its FP32 screening value
};

// How far the FP32 screening vector UBI32.(g32 - c32) of a g can be from its
// exact UBI.g - hkl (c: the box's centre UB.hkl), in the 2-norm: a g of exact
// drlv2 below t^2 has a screening value below (t + margin)^2 (1 + 1e-6).
// Each component of the screened vector is within
//   E = eps S (2 G + W) + 5 eps S |g - c|,  |g - c| <= 2 (G + W),  eps = 2^-24
// of UBI.(g - c): g and c rounded to FP32, then UBI rounded, the difference and
// three roundings of partial sums (S: largest row sum of |UBI|, G: largest |g_j|,
// W: largest half width); 1e-6 covers the FP64 rounding of UB.hkl, as in the
// half widths.  NaN (every g of the cells is evaluated) where FP32 could
// overflow or lose denormals.
__device__ __forceinline__ float screen_margin(const volatile WarpPlan* wp, double G) {
    double S = 0., W = 0.;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        S = fmax(S, fabs(wp->u[3 * r]) + fabs(wp->u[3 * r + 1]) + fabs(wp->u[3 * r + 2]));
        W = fmax(W, wp->w[r]);
    }
    const double E = 5.9604644775390625e-08 * S * (12. * G + 11. * W);
    const double m = kHklMargin + 1.75 * E;  // > sqrt(3) E
    if (!(S < 1e15) || !(G > 1e-15) || !(m < 1e15)) return __int_as_float(0x7fc00000);
    return __double2float_ru(m * (1. + 1e-6));
}

// The screening value from which a g's exact drlv2 cannot be below t^2.
__device__ __forceinline__ float screen_limit(float t, float margin) {
    const float r = t + margin;  // the factor covers its rounding and the squares'
    return r * r * (1.f + 4e-6f);
}

// Evaluate the last `take` waiting candidates (one per lane) in the
// reference's FP64 arithmetic, hand them to act, and drop them from the list.
template <class Act>
__device__ __forceinline__ void eval_candidates(const volatile WarpPlan* wp, Batch* bt, int first,
                                                int take, int lane, const double* __restrict__ gs,
                                                Act& act) {
    const int pos = lane < take ? bt->cp[first + lane] : 0;
    if (lane < take && act.want(pos, bt->cs[first + lane])) {
        double u[9], ih[3], hkl[3];
        const double g[3] = {__ldg(gs + 3 * (int64_t)pos), __ldg(gs + 3 * (int64_t)pos + 1),
                             __ldg(gs + 3 * (int64_t)pos + 2)};
#pragma unroll
        for (int e = 0; e < 9; e++) u[e] = wp->u[e];
        const double sv = drlv2_exact(u, g[0], g[1], g[2], ih);
        unpack_hkl(bt->ch[first + lane], hkl);
        act(pos, sv, ih[0] == hkl[0] && ih[1] == hkl[1] && ih[2] == hkl[2], g, ih);
    }
    __syncwarp();
}

// The g of the listed segments (`total` of them), 32 at a time, screened in
// FP32 against the UBI and the box they were found for; those below the limit
// wait for the FP64 evaluation (whole warps of them are evaluated here; `cn`
// of them wait).  A step's segments are found from the mark bits: the number
// of marks up to a lane's g is its segment.
template <class Act>
__device__ __forceinline__ void scan_segments(const volatile WarpPlan* wp, Batch* bt, int total,
                                              bool last, float limit, int& cn, int lane,
                                              const double* __restrict__ gs,
                                              const float4* __restrict__ g4, Act& act) {
    __syncwarp();  // segments and marks written
    const unsigned le = 0xffffffffu >> (31 - lane);
    int rank0 = -1;
    for (int f0 = 0; f0 < total || last; f0 += 32 * kGAhead) {
        float4 v[kGAhead];
        int pos[kGAhead], box[kGAhead];
#pragma unroll
        for (int q = 0; q < kGAhead; q++) {
            const int word = (f0 >> 5) + q;
            const unsigned mk = word < kMark / 32 ? bt->mark[word] : 0u;
            const int2 sg = bt->seg[max(rank0 + __popc(mk & le), 0)];
            rank0 += __popc(mk);
            const int f = f0 + 32 * q + lane;
            pos[q] = f < total ? f + sg.x : -1;
            box[q] = sg.y;
            if (f < total) v[q] = __ldg(g4 + f + sg.x);
        }
#pragma unroll
        for (int q = 0; q < kGAhead; q++) {
            bool in = false;
            float s = 0.f;
            if (pos[q] >= 0) {
                const float4 c = bt->c[box[q]];
                const float ex = v[q].x - c.x, ey = v[q].y - c.y, ez = v[q].z - c.z;
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    const float d = fmaf(bt->u[3 * r + 2], ez,
                                         fmaf(bt->u[3 * r + 1], ey, bt->u[3 * r] * ex));
                    s = fmaf(d, d, s);
                }
                in = !(s >= limit);
            }
            const unsigned mk = __ballot_sync(0xffffffffu, in);
            if (in) {
                const int slot = cn + __popc(mk & (le >> 1));
                bt->ch[slot] = bt->hkl[box[q]];
                bt->cp[slot] = pos[q];
                bt->cs[slot] = s;
            }
            cn += __popc(mk);
        }
        __syncwarp();
        const bool all = last && f0 + 32 * kGAhead >= total;
        while (cn >= 32 || (all && cn > 0)) {
            const int take = min(cn, 32);
            cn -= take;
            eval_candidates(wp, bt, cn, take, lane, gs, act);
        }
        if (all) break;
    }
    if (lane < kMark / 32) bt->mark[lane] = 0u;
    __syncwarp();
}

// The lookups of `take` queued hkl, one box per lane.  Each lane loads the
// bounds of its box's rows of cells kRowsAhead at a time and lists the rows
// that hold g as segments of one run of g over the warp; when the list is full
// (and after the last row) the run is scanned, so the lanes stay converged
// whatever the boxes' sizes.  Every g within the screen's limit goes to the
// reference's FP64 arithmetic and to act(pos, drlv2, own, g, ih), own = (ih,
// the rounded h, == the box's hkl).  last: the warp's last lookups; the
// candidates still waiting are evaluated too.
//
// Bound: latency of the dependent loads (row bounds, then g) and issue.  The
// g come from the FP32 copy (one 16-byte load instead of three of 8), the
// screen is the ellipsoid's (half the box's volume) and costs FP32
// instructions, and only what passes it is read and evaluated in FP64.  20,000
// UBIs scored at three tolerances over 1.1M g: 6.95 -> 5.64 ms; over 10.2M g at
// one: 11.7 -> 9.9 ms; 2,000 refined over 1.1M g: 0.49 -> 0.37 ms a round.
template <class Act>
__device__ __forceinline__ void lookup_batch(const volatile WarpPlan* wp, Batch* bt,
                                             const unsigned long long* q_w, int take, bool last,
                                             float limit, int& cn, int lane,
                                             const Header* __restrict__ Hp,
                                             const int* __restrict__ start,
                                             const double* __restrict__ gs,
                                             const float4* __restrict__ g4, Act& act) {
    int left = 0, ny = 1, ry = 0, ix1 = 0;
    const int* row = start;  // bounds of the lane's current row, at its first x cell
    const int nx = Hp->nx, nxx = Hp->nxx;
    if (lane < take) {
        Header H;
        H.lo = Hp->lo;
        H.inv_cs = Hp->inv_cs;
        H.inv_csx = Hp->inv_csx;
        H.nx = nx;
        H.nxx = nxx;
        const unsigned long long q = q_w[lane];
        double hkl[3], c[3];
        unpack_hkl(q, hkl);
#pragma unroll
        for (int r = 0; r < 3; r++)
            c[r] = wp->ub[3 * r] * hkl[0] + wp->ub[3 * r + 1] * hkl[1] + wp->ub[3 * r + 2] * hkl[2];
        bt->c[lane] = make_float4(__double2float_rn(c[0]), __double2float_rn(c[1]),
                                  __double2float_rn(c[2]), 0.f);
        bt->hkl[lane] = q;
        const int iy0 = coord(c[1] - wp->w[1], H), iz0 = coord(c[2] - wp->w[2], H);
        const int ix0 = coord_x(c[0] - wp->w[0], H);
        ny = coord(c[1] + wp->w[1], H) - iy0 + 1;
        left = ny * (coord(c[2] + wp->w[2], H) - iz0 + 1);
        ix1 = coord_x(c[0] + wp->w[0], H) + 1 - ix0;
        row = start + ((int64_t)iz0 * nx + iy0) * nxx + ix0;
    }
    int total = 0, nseg = 0;  // listed (uniform)
    int st[kRowsAhead], len[kRowsAhead];
#pragma unroll
    for (int k = 0; k < kRowsAhead; k++) st[k] = len[k] = 0;
    bool have = false;  // rows loaded and not listed yet (uniform)
    for (;;) {
        if (!have) {
            if (__any_sync(0xffffffffu, left > 0)) {
#pragma unroll
                for (int k = 0; k < kRowsAhead; k++) {
                    st[k] = len[k] = 0;
                    if (k < left) {
                        st[k] = __ldg(row);
                        len[k] = __ldg(row + ix1);
                        row += nxx;
                        if (++ry == ny) {
                            ry = 0;
                            row += (int64_t)(nx - ny) * nxx;
                        }
                    }
                }
                left -= kRowsAhead;
#pragma unroll
                for (int k = 0; k < kRowsAhead; k++) len[k] -= st[k];
                have = true;
            }
        }
        bool full = !have;
        if (have) {
            // prefixes of g (low bits) and segments (high bits) over the lanes
            constexpr int kHigh = 24;
            static_assert(32 * kRowsAhead * (kMark + 1) < 1 << kHigh && 32 * kRowsAhead < 256, "");
            unsigned own = 0;
#pragma unroll
            for (int k = 0; k < kRowsAhead; k++)
                own += ((unsigned)(len[k] > 0) << kHigh) + (unsigned)min(len[k], kMark + 1);
            unsigned incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const unsigned all = __shfl_sync(0xffffffffu, incl, 31);
            const int asum = (int)(all & ((1u << kHigh) - 1)), acnt = (int)(all >> kHigh);
            if (acnt <= kSeg - nseg && asum <= kMark - total) {
                int at = total + (int)((incl - own) & ((1u << kHigh) - 1));
                int slot = nseg + (int)((incl - own) >> kHigh);
#pragma unroll
                for (int k = 0; k < kRowsAhead; k++)
                    if (len[k] > 0) {
                        bt->seg[slot++] = make_int2(st[k] - at, lane);
                        if (Act::kPrefetch) asm volatile("prefetch.global.L1 [%0];" ::"l"(g4 + st[k]));
                        atomicOr(bt->mark + (at >> 5), 1u << (at & 31));
                        at += len[k];
                    }
                total += asum;
                nseg += acnt;
                have = false;
            } else if (total > 0) {
                full = true;
            } else {  // more g than the marks hold: the first segment by itself
                const unsigned m = __ballot_sync(0xffffffffu, own > 0);
                const int j = __ffs(m) - 1;
                int n = 0;
                if (lane == j) {
#pragma unroll
                    for (int k = kRowsAhead - 1; k >= 0; k--)
                        if (len[k] > 0) n = len[k];
                    bool first = true;
#pragma unroll
                    for (int k = 0; k < kRowsAhead; k++)
                        if (first && len[k] > 0) {
                            bt->seg[0] = make_int2(st[k], lane);
                            len[k] = 0;
                            first = false;
                        }
                    bt->mark[0] = 1u;
                }
                total = __shfl_sync(0xffffffffu, n, j);
                nseg = 1;
                full = true;
            }
        }
        if (full) {  // the list is full, or the last row is listed
            const bool done = !have;
            if (total > 0 || (done && last))
                scan_segments(wp, bt, total, done && last, limit, cn, lane, gs, g4, act);
            total = nseg = 0;
            if (done) break;
        }
    }
    __syncwarp();
}

// Every (UBI, g) pair of the work item whose drlv2 can be below the plan's
// tolerance (tmax) goes to act(pos, drlv2, own, g, ih): through the hkl lookup
// when ok, else by a plain scan of the regular g (own = true: each g once).
// act.want(pos, s), called first, says whether a g of FP32 screening value s
// (within `margin` of the exact one, screen_margin) is of interest.
template <class Act>
__device__ __forceinline__ void walk(volatile WarpPlan* wp, Batch* bt, unsigned long long* q_w,
                                     bool ok, const Item& it, double tmax, float margin, int lane,
                                     const Header* __restrict__ Hp, int64_t nreg,
                                     const int* __restrict__ start,
                                     const double* __restrict__ gs,
                                     const float4* __restrict__ g4, Act& act) {
    if (!ok) {
        double u[9];
#pragma unroll
        for (int e = 0; e < 9; e++) u[e] = wp->u[e];
        for (int64_t f = (int64_t)it.part * 32 + lane; f < nreg; f += 32 * (int64_t)it.slabs * it.cols) {
            double ih[3];
            const double g[3] = {gs[3 * f], gs[3 * f + 1], gs[3 * f + 2]};
            const double s = drlv2_exact(u, g[0], g[1], g[2], ih);
            act((int)f, s, true, g, ih);
        }
        return;
    }
    int qn = 0, cn = 0;  // hkl queued, candidates waiting (uniform)
    const float limit = screen_limit(__double2float_ru(tmax), margin);
    if (lane < 9) bt->u[lane] = __double2float_rn(wp->u[lane]);
    if (lane < kMark / 32) bt->mark[lane] = 0u;
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
    BoxWalk bw(wp, it);
    for (;;) {
        int h, k, l;
        bool pass;
        const bool more = bw.next(wp, Hp, lane, pass, h, k, l);
        const unsigned mask = __ballot_sync(0xffffffffu, more && pass);
        if (more && pass) q_w[qn + __popc(mask & lt)] = pack_hkl(h, k, l);
        qn += __popc(mask);
        __syncwarp();
        if (qn >= 32 || !more) {
            const int take = min(qn, 32);
            lookup_batch(wp, bt, q_w, take, !more, limit, cn, lane, Hp, start, gs, g4, act);
            const int rest = qn - take;
            unsigned long long v = 0;
            if (lane < rest) v = q_w[32 + lane];
            __syncwarp();
            if (lane < rest) q_w[lane] = v;
            __syncwarp();
            qn = rest;
        }
        if (!more) break;
    }
}

// An act that wants every g the screen lets through.  PREFETCH: a listed row's g are
// brought to L1 while the rest is listed.  Scoring gains by it (20,000 UBIs x 1.1M g
// at three tolerances 5.99 -> 5.66 ms, 112k g 2.75 -> 2.58), refinement and assignment,
// with more to keep in L1, lose 1%.
template <class F, bool PREFETCH = false>
struct EveryG {
    static constexpr bool kPrefetch = PREFETCH;
    F& f;
    __device__ __forceinline__ bool want(int, float) const { return true; }
    __device__ __forceinline__ void operator()(int pos, double s, bool own, const double* g,
                                               const double* ih) const {
        f(pos, s, own, g, ih);
    }
};

// 24 one-warp CTAs per SM (80 registers): 32 spilled 300 bytes a thread.  20,000 UBIs
// at one and three tolerances: 112k g 1.90 -> 1.72 and 2.58 -> 2.30 ms, 1.1M g 2.89 ->
// 2.66 and 5.66 -> 5.64; 20: 1.83, 2.33, 2.79, 5.61.
constexpr int kScoreMinB = 24;

template <int NT>
__global__ void __launch_bounds__(kST, kScoreMinB)
k_score(const double* __restrict__ ubis, int64_t m, Split sp, Header* __restrict__ Hp,
        const int* __restrict__ start, const double* __restrict__ gs,
        const float4* __restrict__ g4, Tols tols,
        int* __restrict__ pcnt, double* __restrict__ psum) {
    __shared__ unsigned long long s_q[kSW][kQueue];
    __shared__ WarpPlan s_plan[kSW];
    __shared__ Batch s_batch[kSW];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t wk = ((int64_t)blockIdx.x * kST + threadIdx.x) >> 5;
    if (wk >= m * sp.parts()) return;  // uniform per warp
    const Item it = sp.item(wk, m);
    const int64_t i = it.i;
    const int64_t nreg = start[Hp->ncells];
    double t2[NT];
    double tmax = 0.;
    int cnt[NT];
    double sum[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        tmax = fmax(tmax, tols.t[j]);
        t2[j] = tols.t[j] * tols.t[j];
        cnt[j] = 0;
        sum[j] = 0.;
    }
    unsigned long long tested = 0;
    const bool ok = setup_plan(s_plan + w, ubis, i, tmax, *Hp, nreg, lane);
    auto count = [&](int, double s, bool own, const double*, const double*) {
        tested++;
        if (own) {
#pragma unroll
            for (int j = 0; j < NT; j++)
                if (s < t2[j]) {
                    cnt[j]++;
                    sum[j] += s;
                }
        }
    };
    EveryG<decltype(count), true> act{count};
    walk(s_plan + w, s_batch + w, s_q[w], ok, it, tmax, screen_margin(s_plan + w, -Hp->lo), lane,
         Hp, nreg, start, gs, g4, act);
    if (!ok && it.part == 0 && lane == 0) atomicAdd(&Hp->nfallback, 1ull);
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const int cs = warp_sum(cnt[j]);
        const double ss = warp_sum(sum[j]);
        if (lane == 0) {
            pcnt[(i * sp.parts() + it.part) * NT + j] = cs;
            psum[(i * sp.parts() + it.part) * NT + j] = ss;
        }
    }
    const long long tt = warp_sum((long long)tested);
    if (lane == 0 && tt) atomicAdd(&Hp->ntested, (unsigned long long)tt);
}

// The g-vectors outside the regular range, one warp per UBI: lanes stride the
// list, fixed-tree warp sums, one slot per UBI and tolerance.
__global__ void __launch_bounds__(kGT)
k_score_special(const double* __restrict__ ubis, int64_t m, int ntol, Tols tols,
                const double* __restrict__ gv, const int* __restrict__ special,
                const int* __restrict__ nspecial, int* __restrict__ scnt,
                double* __restrict__ ssum) {
    const int64_t i = ((int64_t)blockIdx.x * kGT + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= m) return;  // uniform per warp
    int c[ID11B_MAX_TOLS] = {0, 0, 0, 0};
    double sm[ID11B_MAX_TOLS] = {0., 0., 0., 0.};
    const int ns = *nspecial;
    if (ns) {
        double u[9];
        for (int e = 0; e < 9; e++) u[e] = ubis[9 * i + e];
        for (int q = lane; q < ns; q += 32) {
            const int64_t k = special[q];
            double ih[3];
            const double v = drlv2_exact(u, gv[3 * k], gv[3 * k + 1], gv[3 * k + 2], ih);
            for (int j = 0; j < ntol; j++)
                if (v < tols.t[j] * tols.t[j]) {
                    c[j]++;
                    sm[j] += v;
                }
        }
    }
    for (int j = 0; j < ntol; j++) {
        const int cs = warp_sum(c[j]);
        const double ss = warp_sum(sm[j]);
        if (lane == 0) {
            scnt[i * ntol + j] = cs;
            ssum[i * ntol + j] = ss;
        }
    }
}

// One thread per UBI: CTA-part partials in a fixed order, then the slot of
// the g-vectors outside the regular range.
__global__ void __launch_bounds__(kGT)
k_score_finish(int64_t m, int parts, int ntol, const int* __restrict__ pcnt,
               const double* __restrict__ psum, const int* __restrict__ scnt,
               const double* __restrict__ ssum, int* __restrict__ counts,
               double* __restrict__ sums) {
    const int64_t i = (int64_t)blockIdx.x * kGT + threadIdx.x;
    if (i >= m) return;
    int c[ID11B_MAX_TOLS] = {0, 0, 0, 0};
    double s[ID11B_MAX_TOLS] = {0., 0., 0., 0.};
    for (int p = 0; p < parts; p++)
        for (int j = 0; j < ntol; j++) {
            c[j] += pcnt[(i * parts + p) * ntol + j];
            s[j] += psum[(i * parts + p) * ntol + j];
        }
    for (int j = 0; j < ntol; j++) {
        counts[i * ntol + j] = c[j] + scnt[i * ntol + j];
        if (sums) sums[i * ntol + j] = s[j] + ssum[i * ntol + j];
    }
}

// ------------------------------------------------------------ refinement --
// score_and_refine (ImageD11 src/closest.c:267-345) for many UBIs against all
// g through the index: the pairs with drlv2 < tol^2 are exactly the ones the
// lookup hands over with own = true; each adds ih.g^T, ih.ih^T, drlv2 and 1 to
// the normal equations in the reference's FP64 operations, per lane in shared
// memory ([field][lane]), then warp trees, per-part partials and a fixed-order
// finish per UBI that applies the reference's update.
constexpr int kLsqF = 17;  // R 9 (g_i ih_j at 3i+j), H 6 (00 10 20 11 21 22), sum, n

__device__ __forceinline__ void lsq_add(double* acc, double s, const double* g,
                                        const double* ih) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) acc[(3 * i + j) * 32] = dadd(acc[(3 * i + j) * 32], dmul(ih[j], g[i]));
    acc[9 * 32] = dadd(acc[9 * 32], dmul(ih[0], ih[0]));
    acc[10 * 32] = dadd(acc[10 * 32], dmul(ih[1], ih[0]));
    acc[11 * 32] = dadd(acc[11 * 32], dmul(ih[2], ih[0]));
    acc[12 * 32] = dadd(acc[12 * 32], dmul(ih[1], ih[1]));
    acc[13 * 32] = dadd(acc[13 * 32], dmul(ih[2], ih[1]));
    acc[14 * 32] = dadd(acc[14 * 32], dmul(ih[2], ih[2]));
    acc[15 * 32] = dadd(acc[15 * 32], s);
    acc[16 * 32] += 1.0;
}

// (24 CTAs with 80 registers, of which its shared memory, 8.6 KB and 1 KB reserved,
// lets 23 be resident: 2,000 UBIs x 1.1M g 0.42 ms a round; compiled for 32 it
// spills, 0.53 ms)
__global__ void __launch_bounds__(kST, 24)
k_refine(const double* __restrict__ ubis, int64_t m, Split sp, const Header* __restrict__ Hp,
         const int* __restrict__ start, const double* __restrict__ gs,
         const float4* __restrict__ g4, double tol, double* __restrict__ part_out) {
    __shared__ unsigned long long s_q[kSW][kQueue];
    __shared__ WarpPlan s_plan[kSW];
    __shared__ Batch s_batch[kSW];
    __shared__ double s_lsq[kSW][kLsqF * 32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t wk = ((int64_t)blockIdx.x * kST + threadIdx.x) >> 5;
    if (wk >= m * sp.parts()) return;  // uniform per warp
    const Item it = sp.item(wk, m);
    const int64_t i = it.i;
    const int64_t nreg = start[Hp->ncells];
    const double t2 = tol * tol;
    double* acc = s_lsq[w] + lane;
#pragma unroll
    for (int f = 0; f < kLsqF; f++) acc[f * 32] = 0.;
    const bool ok = setup_plan(s_plan + w, ubis, i, tol, *Hp, nreg, lane);
    auto add = [&](int, double s, bool own, const double* g, const double* ih) {
        if (own && s < t2) lsq_add(acc, s, g, ih);
    };
    EveryG<decltype(add)> act{add};
    walk(s_plan + w, s_batch + w, s_q[w], ok, it, tol, screen_margin(s_plan + w, -Hp->lo), lane,
         Hp, nreg, start, gs, g4, act);
    __syncwarp();
#pragma unroll 1
    for (int f = 0; f < kLsqF; f++) {
        const double v = warp_sum(acc[f * 32]);
        if (lane == 0) part_out[(i * sp.parts() + it.part) * kLsqF + f] = v;
    }
}

// One warp per UBI: the items' partials in item order (lane f takes field f), then
// the normal-equation terms of the g outside the regular range (lanes stride the
// list, fixed-tree sums), then the reference's update; n and mean drlv2 of the UBI
// as it was on entry.  Seventeen lanes load an item's row at once: 2,000 UBIs x 10
// items take 5.5 us; 14.5 with one thread per UBI, and 4 for a kernel of its own
// for the list.
__global__ void __launch_bounds__(kGT)
k_refine_finish(double* __restrict__ ubis, int64_t m, int parts,
                const double* __restrict__ part_in, double tol, const double* __restrict__ gv,
                const int* __restrict__ special, const int* __restrict__ nspecial,
                int* __restrict__ npk, double* __restrict__ mean) {
    __shared__ double s_lsq[kGT / 32][kLsqF * 32];
    __shared__ double s_t[kGT / 32][kLsqF];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * kGT + threadIdx.x) >> 5;
    if (i >= m) return;  // uniform per warp
    double t = 0.;
    if (lane < kLsqF) {
        const double* p = part_in + i * parts * kLsqF + lane;
#pragma unroll 4
        for (int q = 0; q < parts; q++) t += p[(int64_t)q * kLsqF];
        s_t[w][lane] = t;
    }
    __syncwarp();
    double u[9];
    for (int e = 0; e < 9; e++) u[e] = ubis[9 * i + e];
    const int ns = *nspecial;
    if (ns) {
        double* acc = s_lsq[w] + lane;
        for (int f = 0; f < kLsqF; f++) acc[f * 32] = 0.;
        for (int q = lane; q < ns; q += 32) {
            const int64_t k = special[q];
            double ih[3];
            const double g[3] = {gv[3 * k], gv[3 * k + 1], gv[3 * k + 2]};
            const double sv = drlv2_exact(u, g[0], g[1], g[2], ih);
            if (sv < tol * tol) lsq_add(acc, sv, g, ih);
        }
        __syncwarp();
        for (int f = 0; f < kLsqF; f++) {
            const double v = warp_sum(acc[f * 32]);
            if (lane == 0) s_t[w][f] += v;
        }
        __syncwarp();
    }
    if (lane != 0) return;
    const double* z = s_t[w];
    double R[9], Hm[9];
    for (int f = 0; f < 9; f++) R[f] = z[f];
    Hm[0] = z[9];  Hm[1] = z[10]; Hm[2] = z[11];
    Hm[3] = z[10]; Hm[4] = z[12]; Hm[5] = z[13];
    Hm[6] = z[11]; Hm[7] = z[13]; Hm[8] = z[14];
    lsq_update_exact(R, Hm, u);
    for (int e = 0; e < 9; e++) ubis[9 * i + e] = u[e];
    const long long n = (long long)z[16];
    if (npk) npk[i] = (int)n;
    if (mean) mean[i] = n > 0 ? z[15] / (double)n : 0.;
}

// ------------------------------------------------------------ assignment --
// Batched score_and_assign (ImageD11 src/closest.c:366-397) over m grains in
// order: for each g the reference's sequence of calls leaves the label of the
// first grain reaching the smallest drlv2 among those below tol^2 and below
// the g's initial drlv2, and that drlv2.  Pass 0 takes the minimum (FP64 bits
// of non-negative values order like the values), pass 1 the lowest grain index
// reaching it; both passes evaluate the same pairs with the same arithmetic.
template <int PASS>
__global__ void __launch_bounds__(kST, ID11B_GRID_MINB)
k_assign(const double* __restrict__ ubis, int64_t m, Split sp, const Header* __restrict__ Hp,
         const int* __restrict__ start, const double* __restrict__ gs,
         const float4* __restrict__ g4, const int* __restrict__ gidx, double tol,
         const double* __restrict__ drlv2,
         unsigned long long* __restrict__ best, int* __restrict__ lab, int64_t base) {
    __shared__ unsigned long long s_q[kSW][kQueue];
    __shared__ WarpPlan s_plan[kSW];
    __shared__ Batch s_batch[kSW];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t wk = ((int64_t)blockIdx.x * kST + threadIdx.x) >> 5;
    if (wk >= m * sp.parts()) return;  // uniform per warp
    const Item it = sp.item(wk, m);
    const int64_t i = it.i;
    const int64_t nreg = start[Hp->ncells];
    const double t2 = tol * tol;
    const bool ok = setup_plan(s_plan + w, ubis, i, tol, *Hp, nreg, lane);
    auto assign = [&](int pos, double s, bool own, const double*, const double*) {
        if (!own || !(s < t2)) return;
        const int k = __ldg(gidx + pos);
        if (!(s < __ldg(drlv2 + k))) return;
        const unsigned long long b = (unsigned long long)__double_as_longlong(s);
        if (PASS == 0)
            atomicMin(best + k, b);
        else if (best[k] == b)
            atomicMin(lab + k, (int)(base + i));
    };
    EveryG<decltype(assign)> act{assign};
    walk(s_plan + w, s_batch + w, s_q[w], ok, it, tol, screen_margin(s_plan + w, -Hp->lo), lane,
         Hp, nreg, start, gs, g4, act);
}

// The same in one pass, for grains that are all here: each g's smallest drlv2
// and the lowest grain reaching it as one 16-byte entry (FP64 bits, grain
// index), lowered by 128-bit compare-and-swap, so that the order of the grains
// does not matter.  Entries are kept by sorted position, next to the g the
// lookups read together, and start at the g's drlv2 on entry (at most tol^2)
// with grain -1: a tie with it does not replace it.
//
// Most pairs below tol^2 lose to a better grain, so each g's current best is
// also kept as a float rounded up (4 bytes: 40 MB for 10M g, in L2), and a
// pair whose FP32 screening value cannot be below it is dropped before its
// FP64 g is read.  The limits only fall, so a stale one drops nothing that
// would win.
//
// Bound: latency and L2 misses of the lookups and the evaluations' random
// reads.  20,000 grains (true ones, 0.2 degrees off) x 10.2M g, tol 0.05: 8.7 ms,
// 9.3 for the whole assignment; the lookup it had before in two passes of atomic
// minima (as k_assign) over every pair, in the caller's g order: 18.8 + 19.1, 38.7 ms.
struct __align__(16) AssignEntry {
    unsigned long long bits;
    long long grain;
};

__device__ __forceinline__ AssignEntry entry_load(const AssignEntry* p) {
    AssignEntry e;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\t"
                 "mov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(e.bits), "=l"(e.grain)
                 : "l"(p)
                 : "memory");
    return e;
}

__device__ __forceinline__ AssignEntry entry_cas(AssignEntry* p, const AssignEntry& was,
                                                 const AssignEntry& now) {
    AssignEntry e;
    asm volatile("{\n\t.reg .b128 t, a, b;\n\tmov.b128 a, {%3, %4};\n\tmov.b128 b, {%5, %6};\n\t"
                 "atom.relaxed.gpu.global.cas.b128 t, [%2], a, b;\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(e.bits), "=l"(e.grain)
                 : "l"(p), "l"(was.bits), "l"(was.grain), "l"(now.bits), "l"(now.grain)
                 : "memory");
    return e;
}

struct AssignAct {
    static constexpr bool kPrefetch = false;
    AssignEntry* entry;
    unsigned* limit;  // float bits, rounded up
    long long grain;
    float margin;

    __device__ __forceinline__ bool want(int pos, float s) const {
        return !(s >= screen_limit(__fsqrt_ru(__uint_as_float(__ldcg(limit + pos))), margin));
    }
    __device__ __forceinline__ void operator()(int pos, double s, bool own, const double*,
                                               const double*) const {
        if (!own || !(s >= 0.)) return;
        const AssignEntry now{(unsigned long long)__double_as_longlong(s), grain};
        AssignEntry was = entry_load(entry + pos);
        while (now.bits < was.bits || (now.bits == was.bits && grain < was.grain)) {
            const AssignEntry got = entry_cas(entry + pos, was, now);
            if (got.bits == was.bits && got.grain == was.grain) {
                atomicMin(limit + pos, __float_as_uint(__double2float_ru(s)));
                break;
            }
            was = got;
        }
    }
};

__global__ void __launch_bounds__(kST, ID11B_GRID_MINB)
k_assign_once(const double* __restrict__ ubis, int64_t m, Split sp,
              const Header* __restrict__ Hp, const int* __restrict__ start,
              const double* __restrict__ gs, const float4* __restrict__ g4, double tol,
              AssignEntry* __restrict__ entry, unsigned* __restrict__ limit) {
    __shared__ unsigned long long s_q[kSW][kQueue];
    __shared__ WarpPlan s_plan[kSW];
    __shared__ Batch s_batch[kSW];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t wk = ((int64_t)blockIdx.x * kST + threadIdx.x) >> 5;
    if (wk >= m * sp.parts()) return;  // uniform per warp
    const Item it = sp.item(wk, m);
    const int64_t nreg = start[Hp->ncells];
    const bool ok = setup_plan(s_plan + w, ubis, it.i, tol, *Hp, nreg, lane);
    const float margin = ok ? screen_margin(s_plan + w, -Hp->lo) : 0.f;
    AssignAct act{entry, limit, (long long)it.i, margin};
    walk(s_plan + w, s_batch + w, s_q[w], ok, it, tol, margin, lane, Hp, nreg, start, gs, g4, act);
}

__global__ void __launch_bounds__(kGT)
k_assign_entries(const int* __restrict__ start, int64_t ncells, const int* __restrict__ gidx,
                 double tol, const double* __restrict__ drlv2, AssignEntry* __restrict__ entry,
                 unsigned* __restrict__ limit) {
    const int64_t nreg = start[ncells];
    const double t2 = tol * tol;
    for (int64_t p = (int64_t)blockIdx.x * kGT + threadIdx.x; p < nreg;
         p += (int64_t)gridDim.x * kGT) {
        const double d = drlv2[gidx[p]];
        const double v = d > 0. ? fmin(d, t2) : 0.;  // NaN and values <= 0: no grain is below
        entry[p] = AssignEntry{(unsigned long long)__double_as_longlong(v), -1};
        limit[p] = __float_as_uint(__double2float_ru(v));
    }
}

constexpr unsigned long long kNoBest = 0x7fffffffffffffffull;

__global__ void __launch_bounds__(kGT)
k_assign_init(int64_t n, unsigned long long* __restrict__ best, int* __restrict__ lab) {
    for (int64_t k = (int64_t)blockIdx.x * kGT + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * kGT) {
        best[k] = kNoBest;  // above the bits of every finite drlv2, and positive as int64
        lab[k] = INT_MAX;
    }
}

// is v one of the grain labels (strictly increasing; null: 0 .. m-1)?
__device__ __forceinline__ bool is_grain_label(int v, const int* __restrict__ gl, int64_t m) {
    if (!gl) return v >= 0 && (int64_t)v < m;
    int64_t lo = 0, hi = m;  // binary search
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        const int x = gl[mid];
        if (x == v) return true;
        if (x < v) lo = mid + 1; else hi = mid;
    }
    return false;
}

// regular g (by sorted position): write the winner, or apply the reference's
// "it does not belong after all" reset when the g held a grain's label
__global__ void __launch_bounds__(kGT)
k_assign_final(const int* __restrict__ start, int64_t ncells, const int* __restrict__ gidx,
               const unsigned long long* __restrict__ best, const int* __restrict__ lab,
               const int* __restrict__ gl, int64_t m, double* __restrict__ drlv2,
               int* __restrict__ labels, int* __restrict__ npk) {
    const int64_t nreg = start[ncells];
    for (int64_t p = (int64_t)blockIdx.x * kGT + threadIdx.x; p < nreg;
         p += (int64_t)gridDim.x * kGT) {
        const int k = gidx[p];
        const int w = lab[k];
        if (w != INT_MAX) {
            labels[k] = gl ? gl[w] : w;
            drlv2[k] = __longlong_as_double((long long)best[k]);
            if (npk) atomicAdd(npk + w, 1);
        } else if (is_grain_label(labels[k], gl, m)) {
            labels[k] = -1;
        }
    }
}

// the same from k_assign_once's entries
__global__ void __launch_bounds__(kGT)
k_assign_winners(const int* __restrict__ start, int64_t ncells, const int* __restrict__ gidx,
                 const AssignEntry* __restrict__ entry, const int* __restrict__ gl, int64_t m,
                 double* __restrict__ drlv2, int* __restrict__ labels, int* __restrict__ npk) {
    const int64_t nreg = start[ncells];
    for (int64_t p = (int64_t)blockIdx.x * kGT + threadIdx.x; p < nreg;
         p += (int64_t)gridDim.x * kGT) {
        const int k = gidx[p];
        const AssignEntry e = entry[p];
        if (e.grain >= 0) {
            labels[k] = gl ? gl[e.grain] : (int)e.grain;
            drlv2[k] = __longlong_as_double((long long)e.bits);
            if (npk) atomicAdd(npk + e.grain, 1);
        } else if (is_grain_label(labels[k], gl, m)) {
            labels[k] = -1;
        }
    }
}

// g outside the regular range: the reference's sequence of calls, literally
__global__ void __launch_bounds__(kGT)
k_assign_special(const double* __restrict__ ubis, int64_t m, const double* __restrict__ gv,
                 const int* __restrict__ spec, const int* __restrict__ nspec, double tol,
                 const int* __restrict__ gl, double* __restrict__ drlv2,
                 int* __restrict__ labels, int* __restrict__ npk) {
    const int ns = *nspec;
    const double t2 = tol * tol;
    for (int q = blockIdx.x * kGT + threadIdx.x; q < ns; q += gridDim.x * kGT) {
        const int64_t k = spec[q];
        const double g0 = gv[3 * k], g1 = gv[3 * k + 1], g2 = gv[3 * k + 2];
        double d = drlv2[k];
        int l = labels[k];
        int64_t win = -1;
        for (int64_t i = 0; i < m; i++) {
            double u[9], ih[3];
            for (int e = 0; e < 9; e++) u[e] = ubis[9 * i + e];
            const double s = drlv2_exact(u, g0, g1, g2, ih);
            const int li = gl ? gl[i] : (int)i;
            if (s < t2 && s < d) {
                l = li;
                d = s;
                win = i;
            } else if (l == li) {
                l = -1;
                win = -1;
            }
        }
        labels[k] = l;
        drlv2[k] = d;
        if (npk && win >= 0) atomicAdd(npk + win, 1);
    }
}

}  // namespace grid
}  // namespace id11b

namespace id11b {
namespace grid {

int num_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
}

unsigned grid_for(int64_t items, int per) {
    int64_t b = (items + per - 1) / per;
    int64_t cap = (int64_t)num_sms() * 8;
    if (b > cap) b = cap;
    return (unsigned)(b > 0 ? b : 1);
}

static int scan_jobs(const ScanJob& a, const ScanJob& b, cudaStream_t st) {
    const unsigned nb = (unsigned)(a.nb + b.nb);
    k_scan_local<<<nb, kScanT, 0, st>>>(a, b);
    ID11B_CHECK_LAUNCH();
    k_scan_totals<<<2, kScanT, 0, st>>>(a, b);
    ID11B_CHECK_LAUNCH();
    k_scan_add<<<nb, kScanT, 0, st>>>(a, b);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

// Work items (warps) per UBI: enough for twice `warps` of them per SM, at least
// `floor`.  More items balance better, but each sets up the UBI's plan and reduces
// its sums.
static int item_parts(int64_t m, int64_t floor, int warps) {
    if (m <= 0) return 1;
    int64_t p = std::max((2 * (int64_t)num_sms() * warps + m - 1) / m, floor);
    return (int)std::min(std::min<int64_t>(p, kMaxParts), INT32_MAX / m);  // one block each
}

static bool few_ubis(int64_t m) { return m < 4 * (int64_t)num_sms() * 64; }

static int64_t index_bytes(int64_t n, int64_t ncells) { return 20 * n + 4 * ncells; }

// An index from which on a second slab (split_for) pays for every UBI's second item,
// however many UBIs there are.  One against two items, us: 20,000 UBIs refined over
// indexes of 34, 45, 53, 58, 59, 73 and 105 MB 2215, 2323, 2773, 3064, 3396, 4201, 6969
// against 2561, 2654, 2835, 3000, 3136, 3607, 5614; 60,000 scored over 13 MB (40,000 of
// them), 59, 70, 82, 105 and 233 MB 3289, 7152, 8867, 11905, 17257, 31497 against 3332,
// 6901, 7882, 10329, 14913, 29055.
constexpr int64_t kTwoSlabs = 56 << 20;

// Scoring: 32 warps an SM (24 are resident).  64, 32 and 24, us: 300 UBIs x 11k, 112k
// and 1.1M g 107, 123, 156; 80, 96, 129; 70, 86, 117 -- 1,000 110, 164, 223; 91, 139, 198;
// 91, 139, 211 -- 3,000 175, 321, 483; 178, 313, 494; 189, 313, 484.  Where there are few
// waves of UBIs two items each: 20,000 x 1.1M at three tolerances 5649 us, 5719 as one.
static int score_parts(int64_t m, int64_t n, int64_t ncells) {
    const bool two = few_ubis(m) || index_bytes(n, ncells) > kTwoSlabs;
    return item_parts(m, two ? 2 : 1, 32);
}

// Assignment, and what a caller's workspace has to hold.
static int least_parts(int64_t m) { return item_parts(m, few_ubis(m) ? 2 : 1, 64); }

// Refinement: an item also reduces 17 sums, so the second is taken only for a slab.
static int refine_parts(int64_t m, int64_t n, int64_t ncells) {
    return item_parts(m, index_bytes(n, ncells) > kTwoSlabs ? 2 : 1, 64);
}

// `parts` work items per UBI as slabs x columns: as many slabs as it takes for a
// slab's FP32 g, row starts and assignment limits to stay in a part of L2 --
// at least `parts` items with `more`, else at most.  32 MB: of a 10.2M-g index
// (250 MB of them), 20,000 grains are assigned in 8.7 ms; one slab 11.8 ms, 96 MB
// 9.9, 48 MB 9.0, 16 MB 9.2, 12 MB 9.3 (each slab goes through every column).  A
// 1.1M-g index (52 MB) is two slabs where there are parts to split.
Split split_for(int parts, bool more, int64_t m, int64_t n, int64_t ncells) {
    int slabs = (int)std::min<int64_t>(16, (index_bytes(n, ncells) + (32 << 20) - 1) >> 25);
    if (slabs < 1) slabs = 1;
    if (!more && slabs > parts) slabs = parts;
    while (slabs > 1 && m > INT32_MAX / (2 * (int64_t)slabs)) slabs--;  // one block per item
    return Split{slabs, more ? (parts + slabs - 1) / slabs : parts / slabs};
}

}  // namespace grid
}  // namespace id11b

using namespace id11b::grid;

extern "C" int id11b_dev_gvec_bounds(const double* gv, int64_t n, uint32_t* bounds, void* stream) {
    if (n < 0 || !bounds || (n > 0 && !gv)) return ID11B_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    ID11B_CHECK(cudaMemsetAsync(bounds, 0, 2 * sizeof(uint32_t), st));
    if (n == 0) return ID11B_OK;
    k_bounds<<<grid_for(n, kGT), kGT, 0, st>>>(gv, n, bounds);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_grid_plan(float gmax, int64_t n, double cell, int32_t* nx, double* cs) {
    if (!nx || !cs || n < 0 || !(gmax >= 0.f) || !(cell >= 0.)) return ID11B_ERR_ARG;
    const double G = (double)gmax * (1. + 1e-6) + 1e-300;
    double c = cell;
    if (c == 0.) c = 2. * G / fmax(1., cbrt((double)n));  // ~one g per cell of the cube
    int64_t k = (int64_t)ceil(2. * G / c);
    if (k < 1) k = 1;
    if (k > 400) {  // at most 6.4e7 cells
        k = 400;
    }
    *nx = (int32_t)k;
    *cs = fmax(c, 2. * G / (double)k);
    return ID11B_OK;
}

namespace id11b {
namespace grid {
bool grid_dims_ok(int32_t nx, int32_t xsub) {
    return nx >= 1 && nx <= 400 && xsub >= 1 && xsub <= 16 && (int64_t)nx * nx * nx * xsub <= (1 << 26);
}
}  // namespace grid
}  // namespace id11b

extern "C" int64_t id11b_grid_bytes(int64_t n, int32_t nx, int32_t xsub) {
    if (n < 0 || !grid_dims_ok(nx, xsub)) return -1;
    return (int64_t)layout(n, (int64_t)nx * nx * nx * xsub).bytes;
}

extern "C" int id11b_dev_build_grid(const double* gv, int64_t n, float gmax, float rmax, double cs,
                                    int32_t nx, int32_t xsub, void* gridbuf, int64_t grid_bytes,
                                    void* stream) {
    if (n < 0 || !grid_dims_ok(nx, xsub) || !gridbuf || (n > 0 && !gv) || !(cs > 0.) ||
        !(gmax >= 0.f) || !(rmax >= 0.f))
        return ID11B_ERR_ARG;
    if ((uintptr_t)gridbuf & 255) return ID11B_ERR_ALIGN;
    if (n > INT32_MAX - 1) return ID11B_ERR_SIZE;
    const int64_t ncells = (int64_t)nx * nx * nx * xsub;
    const Layout L = layout(n, ncells);
    if (grid_bytes < (int64_t)L.bytes) return ID11B_ERR_SIZE;
    cudaStream_t st = (cudaStream_t)stream;
    char* b = (char*)gridbuf;
    Header h;
    memset(&h, 0, sizeof(h));
    h.lo = -((double)gmax * (1. + 1e-6) + 1e-300);
    h.cs = cs;
    h.inv_cs = 1.0 / cs;
    h.inv_csx = (double)xsub / cs;
    h.rmax = (double)rmax;
    h.ncells = ncells;
    h.n = n;
    h.nx = nx;
    h.nxx = nx * xsub;
    static_assert(sizeof(Header) <= 256, "header");
    int* cnt = (int*)(b + L.cnt);
    int* start = (int*)(b + L.start);
    int* flag = (int*)(b + L.flag);
    int* spos = (int*)(b + L.spos);
    int* tot = (int*)(b + L.tot);
    int* place = (int*)(b + L.g4);  // until k_place writes g4
    Header* H = (Header*)(b + L.header);
    ID11B_CHECK(cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)(ncells + 1), st));
    k_count<<<grid_for(n, kGT), kGT, 0, st>>>(gv, n, h, H, cnt, flag, place);
    ID11B_CHECK_LAUNCH();
    const int cb = (int)scan_blocks(ncells + 1);
    const int rc = scan_jobs(ScanJob{cnt, ncells + 1, start, tot, cb},
                             ScanJob{flag, n + 1, spos, tot + cb, (int)scan_blocks(n + 1)}, st);
    if (rc || n == 0) return rc;
    int* list = flag;  // the flags are done with
    k_list_cells<<<grid_for(n, kGT), kGT, 0, st>>>(gv, n, H, start, place, list, spos,
                                                   (int*)(b + L.spec));
    ID11B_CHECK_LAUNCH();
    k_place<<<grid_for(n, kGT), kGT, 0, st>>>(gv, H, start, list, (double*)(b + L.g),
                                              (int*)(b + L.idx), (float4*)(b + L.g4));
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

// partials: (m * parts + m) x ntol ints, then the same doubles (the last m x
// ntol of each: the g outside the regular range)
static int64_t score_bytes(int64_t m, int ntol, int parts) {
    const int64_t mm = m > 0 ? m : 1;
    const int64_t items = (mm * parts + mm) * ntol;
    return (int64_t)(al256(sizeof(int) * (size_t)items) + al256(sizeof(double) * (size_t)items));
}

// room for two items per UBI; a call takes one where the workspace has no more
extern "C" int64_t id11b_grid_score_workspace_bytes(int64_t m, int ntol) {
    if (m < 0 || ntol < 1 || ntol > ID11B_MAX_TOLS) return -1;
    return score_bytes(m, ntol, std::max(least_parts(m), 2));
}

extern "C" int id11b_dev_score_grid(const double* ubis, int64_t m, const double* gv, int64_t n,
                                    int32_t nx, int32_t xsub, const void* gridbuf,
                                    const double* tols_host, int ntol, int32_t* counts,
                                    double* sums, void* ws, int64_t ws_bytes, void* stream) {
    if (!tols_host || ntol < 1 || ntol > ID11B_MAX_TOLS || m < 0 || n < 0 ||
        !grid_dims_ok(nx, xsub) || !gridbuf || !ws || (m > 0 && (!ubis || !counts)) ||
        (n > 0 && !gv))
        return ID11B_ERR_ARG;
    Tols T;
    T.fix = 0.;  // the lookup's sums are fixed-order FP64
    for (int j = 0; j < ID11B_MAX_TOLS; j++) T.t[j] = j < ntol ? tols_host[j] : 0.;
    for (int j = 0; j < ntol; j++)
        if (!(tols_host[j] >= 0.) || !(tols_host[j] < 1e3)) return ID11B_ERR_ARG;
    if (((uintptr_t)gridbuf & 255) || ((uintptr_t)ws & 255)) return ID11B_ERR_ALIGN;
    if (ws_bytes < score_bytes(m, ntol, least_parts(m))) return ID11B_ERR_SIZE;
    if (m > INT32_MAX) return ID11B_ERR_SIZE;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t ncells = (int64_t)nx * nx * nx * xsub;
    const Layout L = layout(n, ncells);
    char* b = (char*)gridbuf;
    Header* H = (Header*)b;
    ID11B_CHECK(cudaMemsetAsync(&H->nfallback, 0, 3 * sizeof(unsigned long long), st));
    if (m == 0) return ID11B_OK;
    int parts = score_parts(m, n, ncells);
    if (score_bytes(m, ntol, parts) > ws_bytes) parts = 1;
    const int64_t items = (m * parts + m) * ntol;
    int* pcnt = (int*)ws;
    double* psum = (double*)((char*)ws + al256(sizeof(int) * (size_t)items));
    int* scnt = pcnt + m * parts * ntol;
    double* ssum = psum + m * parts * ntol;
    const Split sp = split_for(parts, false, m, n, ncells);
    const unsigned blocks = (unsigned)((m * sp.parts() + kSW - 1) / kSW);
    const int* start = (const int*)(b + L.start);
    const double* gs = (const double*)(b + L.g);
    const float4* g4 = (const float4*)(b + L.g4);
    switch (ntol) {
        case 1: k_score<1><<<blocks, kST, 0, st>>>(ubis, m, sp, H, start, gs, g4, T, pcnt, psum); break;
        case 2: k_score<2><<<blocks, kST, 0, st>>>(ubis, m, sp, H, start, gs, g4, T, pcnt, psum); break;
        case 3: k_score<3><<<blocks, kST, 0, st>>>(ubis, m, sp, H, start, gs, g4, T, pcnt, psum); break;
        default: k_score<4><<<blocks, kST, 0, st>>>(ubis, m, sp, H, start, gs, g4, T, pcnt, psum); break;
    }
    ID11B_CHECK_LAUNCH();
    k_score_special<<<(unsigned)((m * 32 + kGT - 1) / kGT), kGT, 0, st>>>(
        ubis, m, ntol, T, gv, (const int*)(b + L.spec), (const int*)(b + L.spos) + n, scnt,
        ssum);
    ID11B_CHECK_LAUNCH();
    k_score_finish<<<(unsigned)((m + kGT - 1) / kGT), kGT, 0, st>>>(m, sp.parts(), ntol, pcnt, psum,
                                                                    scnt, ssum, counts, sums);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_grid_stats(const void* gridbuf, int64_t* nregular, int64_t* nspecial,
                                int64_t* nfallback, int64_t* ntested, int64_t* npairs,
                                void* stream) {
    if (!gridbuf) return ID11B_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    Header h;
    ID11B_CHECK(cudaMemcpyAsync(&h, gridbuf, sizeof(h), cudaMemcpyDeviceToHost, st));
    ID11B_CHECK(cudaStreamSynchronize(st));
    const Layout L = layout(h.n, h.ncells);
    int nr = 0, ns = 0;
    ID11B_CHECK(cudaMemcpyAsync(&nr, (const char*)gridbuf + L.start + sizeof(int) * h.ncells,
                                sizeof(int), cudaMemcpyDeviceToHost, st));
    ID11B_CHECK(cudaMemcpyAsync(&ns, (const char*)gridbuf + L.spos + sizeof(int) * h.n,
                                sizeof(int), cudaMemcpyDeviceToHost, st));
    ID11B_CHECK(cudaStreamSynchronize(st));
    if (nregular) *nregular = nr;
    if (nspecial) *nspecial = ns;
    if (nfallback) *nfallback = (int64_t)h.nfallback;
    if (ntested) *ntested = (int64_t)h.ntested;
    if (npairs) *npairs = (int64_t)h.npairs;
    return ID11B_OK;
}

// entries (16 bytes) and limits (4) per g
extern "C" int64_t id11b_assign_workspace_bytes(int64_t n) {
    if (n < 0) return -1;
    const size_t nn = (size_t)(n > 0 ? n : 1);
    return (int64_t)(al256(sizeof(AssignEntry) * nn) + al256(sizeof(unsigned) * nn));
}

extern "C" int id11b_dev_score_and_assign_grid(const double* ubis, int64_t m,
                                               const int32_t* grain_labels, const double* gv,
                                               int64_t n, int32_t nx, int32_t xsub,
                                               const void* gridbuf, double tol, double* drlv2,
                                               int32_t* labels, int32_t* npk, void* ws,
                                               int64_t ws_bytes, void* stream) {
    if (m < 0 || n < 0 || !grid_dims_ok(nx, xsub) || !gridbuf || !ws || (m > 0 && !ubis) ||
        (n > 0 && (!gv || !drlv2 || !labels)) || !(tol >= 0.) || !(tol < 1e3))
        return ID11B_ERR_ARG;
    if (((uintptr_t)gridbuf & 255) || ((uintptr_t)ws & 255)) return ID11B_ERR_ALIGN;
    if (ws_bytes < id11b_assign_workspace_bytes(n)) return ID11B_ERR_SIZE;
    if (m > INT32_MAX - 1) return ID11B_ERR_SIZE;
    cudaStream_t st = (cudaStream_t)stream;
    if (npk && m > 0) ID11B_CHECK(cudaMemsetAsync(npk, 0, sizeof(int32_t) * (size_t)m, st));
    if (m == 0 || n == 0) return ID11B_OK;
    const int64_t ncells = (int64_t)nx * nx * nx * xsub;
    const Layout L = layout(n, ncells);
    const char* b = (const char*)gridbuf;
    const Header* H = (const Header*)b;
    const int* start = (const int*)(b + L.start);
    const int* gidx = (const int*)(b + L.idx);
    AssignEntry* entry = (AssignEntry*)ws;
    unsigned* limit = (unsigned*)((char*)ws + al256(sizeof(AssignEntry) * (size_t)n));
    k_assign_entries<<<grid_for(n, kGT), kGT, 0, st>>>(start, ncells, gidx, tol, drlv2, entry,
                                                       limit);
    ID11B_CHECK_LAUNCH();
    const Split sp = split_for(least_parts(m), true, m, n, ncells);
    k_assign_once<<<(unsigned)((m * sp.parts() + kSW - 1) / kSW), kST, 0, st>>>(
        ubis, m, sp, H, start, (const double*)(b + L.g), (const float4*)(b + L.g4), tol, entry,
        limit);
    ID11B_CHECK_LAUNCH();
    k_assign_winners<<<grid_for(n, kGT), kGT, 0, st>>>(start, ncells, gidx, entry, grain_labels, m,
                                                       drlv2, labels, npk);
    ID11B_CHECK_LAUNCH();
    k_assign_special<<<grid_for(n, kGT), kGT, 0, st>>>(ubis, m, gv, (const int*)(b + L.spec),
                                                       (const int*)(b + L.spos) + n, tol,
                                                       grain_labels, drlv2, labels, npk);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

// partials: 17 doubles per work item (the same two sizes as scoring)
static int64_t refine_bytes(int64_t m, int parts) {
    return (int64_t)al256(sizeof(double) * kLsqF * (size_t)(m > 0 ? m : 1) * parts);
}

extern "C" int64_t id11b_grid_refine_workspace_bytes(int64_t m) {
    if (m < 0) return -1;
    return refine_bytes(m, std::max(least_parts(m), 2));
}

extern "C" int id11b_dev_refine_grid(double* ubis, int64_t m, const double* gv, int64_t n,
                                     int32_t nx, int32_t xsub, const void* gridbuf, double tol,
                                     int iters, int32_t* npk, double* mean, void* ws,
                                     int64_t ws_bytes, void* stream) {
    if (m < 0 || n < 0 || iters < 0 || !grid_dims_ok(nx, xsub) || !gridbuf || !ws ||
        (m > 0 && !ubis) || (n > 0 && !gv) || !(tol >= 0.) || !(tol < 1e3))
        return ID11B_ERR_ARG;
    if (((uintptr_t)gridbuf & 255) || ((uintptr_t)ws & 255)) return ID11B_ERR_ALIGN;
    if (ws_bytes < refine_bytes(m, least_parts(m))) return ID11B_ERR_SIZE;
    if (m > INT32_MAX) return ID11B_ERR_SIZE;
    cudaStream_t st = (cudaStream_t)stream;
    if (m == 0) return ID11B_OK;
    const Layout L = layout(n, (int64_t)nx * nx * nx * xsub);
    const char* b = (const char*)gridbuf;
    const Header* H = (const Header*)b;
    const int64_t ncells = (int64_t)nx * nx * nx * xsub;
    int parts = refine_parts(m, n, ncells);
    if (refine_bytes(m, parts) > ws_bytes) parts = 1;
    const Split sp = split_for(parts, false, m, n, ncells);
    const unsigned blocks = (unsigned)((m * sp.parts() + kSW - 1) / kSW);
    double* part = (double*)ws;
    for (int it = 0; it < iters; it++) {
        k_refine<<<blocks, kST, 0, st>>>(ubis, m, sp, H, (const int*)(b + L.start),
                                         (const double*)(b + L.g), (const float4*)(b + L.g4), tol,
                                         part);
        ID11B_CHECK_LAUNCH();
        k_refine_finish<<<(unsigned)((m * 32 + kGT - 1) / kGT), kGT, 0, st>>>(
            ubis, m, sp.parts(), part, tol, gv, (const int*)(b + L.spec),
            (const int*)(b + L.spos) + n, npk, mean);
        ID11B_CHECK_LAUNCH();
    }
    return ID11B_OK;
}

// The assignment in pieces, for grains sharded over ranks: every rank runs
// pass -1 (reset) and pass 0 over its share of the grains, the best arrays are
// reduced with MIN over ranks (int64 view), pass 1 over the share, the lab
// arrays reduced with MIN (int32), and every rank then applies
// id11b_dev_assign_grid_final with all m grains (for the g outside the
// regular range, which follow the reference's sequence of calls).
extern "C" int id11b_dev_assign_grid_pass(const double* ubis, int64_t m, int64_t index_base,
                                          int64_t n, int32_t nx, int32_t xsub,
                                          const void* gridbuf, double tol, const double* drlv2,
                                          int pass, uint64_t* best, int32_t* lab, void* stream) {
    if (m < 0 || n < 0 || index_base < 0 || index_base + m > INT32_MAX - 1 ||
        !grid_dims_ok(nx, xsub) || !gridbuf || !best || !lab || (m > 0 && !ubis) ||
        (n > 0 && !drlv2) || !(tol >= 0.) || !(tol < 1e3) || pass < -1 || pass > 1)
        return ID11B_ERR_ARG;
    if ((uintptr_t)gridbuf & 255) return ID11B_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    if (n == 0) return ID11B_OK;
    if (pass == -1) {
        k_assign_init<<<grid_for(n, kGT), kGT, 0, st>>>(n, (unsigned long long*)best, lab);
        ID11B_CHECK_LAUNCH();
        return ID11B_OK;
    }
    if (m == 0) return ID11B_OK;
    const Layout L = layout(n, (int64_t)nx * nx * nx * xsub);
    const char* b = (const char*)gridbuf;
    const Split sp = split_for(least_parts(m), true, m, n, (int64_t)nx * nx * nx * xsub);
    const unsigned blocks = (unsigned)((m * sp.parts() + kSW - 1) / kSW);
    if (pass == 0)
        k_assign<0><<<blocks, kST, 0, st>>>(ubis, m, sp, (const Header*)b,
                                            (const int*)(b + L.start), (const double*)(b + L.g),
                                            (const float4*)(b + L.g4), (const int*)(b + L.idx),
                                            tol, drlv2,
                                            (unsigned long long*)best, lab, index_base);
    else
        k_assign<1><<<blocks, kST, 0, st>>>(ubis, m, sp, (const Header*)b,
                                            (const int*)(b + L.start), (const double*)(b + L.g),
                                            (const float4*)(b + L.g4), (const int*)(b + L.idx),
                                            tol, drlv2,
                                            (unsigned long long*)best, lab, index_base);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}

extern "C" int id11b_dev_assign_grid_final(const double* ubis, int64_t m,
                                           const int32_t* grain_labels, const double* gv,
                                           int64_t n, int32_t nx, int32_t xsub,
                                           const void* gridbuf, double tol, const uint64_t* best,
                                           const int32_t* lab, double* drlv2, int32_t* labels,
                                           int32_t* npk, void* stream) {
    if (m < 0 || n < 0 || !grid_dims_ok(nx, xsub) || !gridbuf || !best || !lab ||
        (m > 0 && !ubis) || (n > 0 && (!gv || !drlv2 || !labels)) || !(tol >= 0.) ||
        !(tol < 1e3) || m > INT32_MAX - 1)
        return ID11B_ERR_ARG;
    if ((uintptr_t)gridbuf & 255) return ID11B_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    if (npk && m > 0) ID11B_CHECK(cudaMemsetAsync(npk, 0, sizeof(int32_t) * (size_t)m, st));
    if (m == 0 || n == 0) return ID11B_OK;
    const int64_t ncells = (int64_t)nx * nx * nx * xsub;
    const Layout L = layout(n, ncells);
    const char* b = (const char*)gridbuf;
    k_assign_final<<<grid_for(n, kGT), kGT, 0, st>>>(
        (const int*)(b + L.start), ncells, (const int*)(b + L.idx),
        (const unsigned long long*)best, lab, grain_labels, m, drlv2, labels, npk);
    ID11B_CHECK_LAUNCH();
    k_assign_special<<<grid_for(n, kGT), kGT, 0, st>>>(ubis, m, gv, (const int*)(b + L.spec),
                                                       (const int*)(b + L.spos) + n, tol,
                                                       grain_labels, drlv2, labels, npk);
    ID11B_CHECK_LAUNCH();
    return ID11B_OK;
}
