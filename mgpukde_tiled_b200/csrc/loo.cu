// Leave-one-out log likelihood for a list of bandwidths in one launch.
//
// LogLikelihood (kde_cuda_kdtr_tiled.cu:3214-3299) recomputes the edge
// weights at h, scatters K_h(d) w_i e_i into every neighbour of i found by a
// k-d tree range search (DensityAtPointsKdtr, kde_kernel_kdtr.cu:681-804),
// subtracts the self term and takes logf(max(den, EPSILONDENSITY))
// (dCopyDensityValues, :806-830), then sums in float (ReductionSum,
// :1045-1111); MLE_FixedBandWidth (:3044-3093) calls it twice per
// golden-section step.  Here the density at query point j is gathered over
// its neighbours i != j:
//   loo_j(h) = sum_{i != j, d^2 < 9h^2} exp(-d^2 / 2h^2) / (h^2 TWO_PI) w_i e_i(h)
//   logL(h)  = sum_j log(max(loo_j(h), EPSILONDENSITY))
// for every h of a list, as one persistent launch over work items
// (h, group of 128 queries, quarter of the group[, part of its candidates]),
// one warp each, heaviest h first, fed from a global item counter.  The points
// are indexed once per bandwidth octave (row-major bins of side in (0.375 h,
// 0.75 h] for the h that use the level), so the candidates of a group are one
// contiguous range per bin row.  A group is 128 consecutive records of the
// Z-order of the bins.  Candidates come in batches of 64, two per lane, into
// the warp's shared memory; every lane (one query) scans them, two candidates
// at a time in packed FP32.  The cutoff is decided in FP32 with a band around
// 9h^2 re-decided by the oracle's exact FP64 test, so the summed pair set is
// exactly the oracle's; terms are FP32 (an exp2 by range reduction and a
// polynomial, free of the systematic bias an approximate special-function
// exp2 would add to every one of the sum's terms), summed over at most 128
// candidates of one bin row and added into a Kahan-compensated FP32
// accumulator; the per-query log is FP64, and the per-group and per-h sums are
// fixed-order FP64 trees (bitwise reproducible).  The argmax is taken on the
// device.  The whole sequence (edge weights for every h, the gather, the
// sums, the argmax) is captured once into a CUDA graph and replayed, with the
// bandwidths read from device memory, so a golden-section step is one graph
// launch.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <vector>

#include "mgk_internal.cuh"

namespace {

constexpr int kLooQ = 128;    // queries of a group; a work item is a quarter of one, a query per lane
constexpr int kLooSub = kLooQ / 32;
constexpr int kLooB = 64;     // candidates per staged batch, two per lane
constexpr int kLooSum = 128;  // candidates of a bin row summed in plain FP32 before each Kahan step
constexpr int kLooWarps = 4;  // warps per CTA, each with work items of its own
constexpr int kMaxLev = 16;   // bandwidth octaves
constexpr int kMaxSplit = 16;
constexpr unsigned kMaxGridY = 65535;  // longer lists of bandwidths go through it again
constexpr int64_t kMaxItems = 1ll << 31;  // work items of a launch (32-bit numbers, handed out past the last)
// candidates of a batch scanned at a time (one test for the rare cases)
#ifndef MGK_LOO_TRIP
#define MGK_LOO_TRIP 8
#endif
constexpr int kLooTrip = MGK_LOO_TRIP;
static_assert(kLooB % kLooTrip == 0 && kLooTrip % 2 == 0 && kLooSum % kLooTrip == 0, "whole trips");

struct LevelDesc {
    const MgkPt* pts;
    const int32_t* bin_start;
    const int32_t* perm;
    const int32_t* qord;  // query order: record positions in Z-order of the bins
    double ox, oy, side, inv_side;
    int64_t nbx, nby;
};

struct LooParams {
    const LevelDesc* lev;  // [nlev], device
    double side[kMaxLev];  // bin side of each level
    int nlev;
    int nsplit;  // parts of a group's candidates, each a work item of its own
    int64_t n;
    int g0, gcount;       // this share's query groups [g0, g0 + gcount) (all groups: from 0)
    int nh;
    int k0, k1;           // places in the processing order that a launch of the scan takes
    const float* hgrid;   // [nh]
    int* korder;          // [nh] processing order (largest h first)
    int* klevel;          // [nh] level of each h
    // edge weights, or null (no edge correction): e_i(h_k) of point i (input
    // order) is ew[(i / ew_chunk) * ew_cstride + k * ew_chunk + i % ew_chunk],
    // i.e. chunks of ew_chunk points, each nh rows of ew_chunk floats (one
    // chunk of n points, [nh][n], in a single-process batch)
    const float* ew;
    int64_t ew_chunk, ew_cstride;
    // w e of every record of the level that h_k uses, in record order ([nh][n]), or null
    float* wl;
    double* psum;         // [nsplit][nh][gcount * kLooSub][32] unnormalised sums (nsplit > 1), else null
    double* part;         // [nh][gcount * kLooSub]
    unsigned* counter;    // [0] work-item queue head, [1] finished bandwidths
    unsigned long long* evals;  // pairs; the edge cells' count lies before it
};

// What the host gives a run and gets from it, in mapped memory (device
// addresses), so that no copy goes through a copy engine: four copies, two
// memsets, a kernel for the argmax and page-locked buffers made per batch took
// 30 us of a batch and 15 us of each golden-section step (16 bandwidths on
// 2,000 points 278 -> 250 us, a search on 20,000 points 3.31 -> 3.13 ms, on
// 1,000 1.22 -> 1.05 ms).
struct LooHost {
    const float* h;        // [nh]
    const LevelDesc* lev;  // [nlev]
    double* logl;          // [nh]
    unsigned long long* evals;  // edge cells, pairs
    int* best;
};

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The log of a query's leave-one-out density from its unnormalised sum.
__device__ __forceinline__ double loo_log(double sum, double h2) {
    const double loo = sum / (h2 * (double)MGK_TWO_PI_F);
    const double fl = (double)MGK_EPS_DENSITY_F;
    return log(loo > fl ? loo : fl);
}

// The run's bandwidths and the levels into device memory, the counters to
// zero; level and processing order of every h (one CTA; nh is small).
__global__ void k_loo_prep(LooParams P, LooHost H, float* hgrid, LevelDesc* __restrict__ lev) {  // hgrid is P.hgrid
    for (int k = threadIdx.x; k < P.nh; k += blockDim.x) hgrid[k] = H.h[k];
    for (int l = threadIdx.x; l < P.nlev; l += blockDim.x) lev[l] = H.lev[l];
    if (threadIdx.x < 2) {
        P.counter[threadIdx.x] = 0u;
        P.evals[(int)threadIdx.x - 1] = 0ull;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < P.nh; k += blockDim.x) {
        const float h = P.hgrid[k];
        int L = 0;
        for (int l = 1; l < P.nlev; l++)
            if (P.side[l] <= 0.75 * (double)h) L = l;
        int rank = 0;
        for (int j = 0; j < P.nh; j++) {
            const float hj = P.hgrid[j];
            rank += (hj > h) || (hj == h && j < k);
        }
        P.klevel[k] = L;
        P.korder[rank] = k;
    }
}

// wl[k][i] = w e(h_k) of record i of the level of h_k: the scan then reads its
// candidates' weights in order instead of through the permutation.
__global__ void k_loo_weights(LooParams P) {
    for (int k = blockIdx.y; k < P.nh; k += gridDim.y) {
        const LevelDesc L = P.lev[P.klevel[k]];
        const float* ewk = P.ew + (int64_t)k * P.ew_chunk;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < P.n; i += (int64_t)gridDim.x * blockDim.x) {
            const int64_t pi = L.perm[i], ch = pi / P.ew_chunk;
            P.wl[(int64_t)k * P.n + i] = L.pts[i].wk * ewk[ch * P.ew_cstride + (pi - ch * P.ew_chunk)];
        }
    }
}

// What bounds it: the issue slots and the FMA pipe together (about 23
// instructions and 21 FMA-pipe cycles per candidate and warp; ncu: 73 % of the
// issue slots, 68 % of the FMA cycles).  200,000 points, 64 bandwidths in
// [5, 500]: 225 ms before (scalar FP32, 128 queries a CTA between two
// barriers per batch, 1.72 tests per pair), 125 ms now.  What gave it:
//  - distances, exponents and range reduction two candidates at a time (f32x2);
//  - the polynomial scalar, its coefficients immediates (see mgk_exp2_neg_frac);
//  - pair counts from sign bits: a predicated increment costs two instructions;
//  - a warp its own work item: no CTA barriers, and rows cut to the disc
//    around 32 queries instead of the square around 128 (1.38 tests a pair).
// Finer bins or a Hilbert order would cut the tests to 1.2 a pair, but then
// the pieces summed in plain FP32 hold other candidates, and with edge weights
// of points outside the study area (10^6 and more) logL moves by 3e-9.
// More resident warps (80 or 64 registers) spill and are slower: 134 ms.
// Resident CTAs per SM that bound the registers.
#ifndef MGK_LOO_MIN_CTAS
#define MGK_LOO_MIN_CTAS 4
#endif

__global__ void __launch_bounds__(kLooWarps * 32, MGK_LOO_MIN_CTAS) k_loo_multi(LooParams P) {
    // per warp: candidates by component (xh, yh, xl, yl, weight), two batches
    __shared__ __align__(16) float s_cand[kLooWarps][2][5][kLooB];
    // of the window's rows: their slots end, what takes a slot to its place in
    // the group's range of the row, that range's first record, the place where
    // this item's part of it ends
    __shared__ int4 s_row[kLooWarps][32];
    const int warp = threadIdx.x >> 5;
    int lane;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));  // kept in a register
    float(*cand)[5][kLooB] = s_cand[warp];
    int4* row = s_row[warp];
    const unsigned ngs = (unsigned)P.gcount * kLooSub;  // quarters of groups
    const unsigned per_h = ngs * (unsigned)P.nsplit;
    const unsigned total = (unsigned)(P.k1 - P.k0) * per_h;
    const f2 magic = f2_dup(12582912.0f);  // 1.5 2^23: adding it rounds to the nearest integer
    unsigned long long cnt_all = 0;
    for (;;) {
        unsigned item = 0;
        if (lane == 0) item = atomicAdd(P.counter, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= total) break;
        const int k = P.korder[P.k0 + (int)(item / per_h)];
        const int split = (int)((item % per_h) / ngs);
        const int gi = (int)((item % per_h) % ngs);  // quarter gi % kLooSub of group gi / kLooSub
        const LevelDesc& L = P.lev[P.klevel[k]];
        const float h = P.hgrid[k];
        const double h2 = mgk_h2(h);
        const double cut = MGK_CUT * h2;
        const float cutf = (float)cut;
        const float epsd2 = cutf * 4e-6f;
        // log2(e) / (2 h^2) as a float pair: a one-float scale would bias every
        // exponent of the batch the same way
        const double k2 = MGK_LOG2E / (2.0 * h2);
        const float k2h = (float)k2, k2l = (float)(k2 - (double)k2h);
        const double reach = sqrt(cut) * (1.0 + 1e-9);
        const MgkPt* __restrict__ pts = L.pts;
        const float* __restrict__ wl = P.wl ? P.wl + (int64_t)k * P.n : nullptr;

        // this lane's query, and the bounding boxes of the item's queries and of the group's
        const int64_t q0 = (int64_t)(P.g0 + gi / kLooSub) * kLooQ;
        int qpos = -1;
        float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float mnx = FLT_MAX, mxx = -FLT_MAX, mny = FLT_MAX, mxy = -FLT_MAX;
        float gmnx = FLT_MAX, gmxx = -FLT_MAX;
#pragma unroll
        for (int i = 0; i < kLooSub; i++) {
            const int64_t qk = q0 + 32 * i + lane;
            if (qk >= P.n) continue;
            const int qp = L.qord[qk];
            const float4 v = *reinterpret_cast<const float4*>(pts + qp);
            const float vx = v.x + v.z, vy = v.y + v.w;
            gmnx = fminf(gmnx, vx);
            gmxx = fmaxf(gmxx, vx);
            if (i == gi % kLooSub) {
                q = v;
                qpos = qp;
                mnx = mxx = vx;
                mny = mxy = vy;
            }
        }
        const bool qv = qpos >= 0;
        const float qx = q.x + q.z, qy = q.y + q.w;
        for (int o = 16; o; o >>= 1) {
            mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
            mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
            mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
            mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
            gmnx = fminf(gmnx, __shfl_xor_sync(0xffffffffu, gmnx, o));
            gmxx = fmaxf(gmxx, __shfl_xor_sync(0xffffffffu, gmxx, o));
        }
        if (mnx > mxx) {  // no query in this quarter
            if (P.psum) P.psum[(((int64_t)split * P.nh + k) * ngs + gi) * 32 + lane] = 0.0;
            else if (lane == 0) P.part[(int64_t)k * ngs + gi] = 0.0;
            continue;
        }
        const int by0 = (int)fmax(0.0, floor(((double)mny - reach - L.oy) * L.inv_side));
        const int by1 = (int)fmin((double)(L.nby - 1), floor(((double)mxy + reach - L.oy) * L.inv_side));
        // the group's bin columns
        const double g0 = fmax(0.0, floor(((double)gmnx - reach - L.ox) * L.inv_side));
        const double g1 = fmin((double)(L.nbx - 1), floor(((double)gmxx + reach - L.ox) * L.inv_side));
        // the query's bin row, as the index assigns it
        const int qby = (int)fmin(fmax(floor(((double)qy - L.oy) * L.inv_side), 0.0), (double)(L.nby - 1));

        const f2 qxh = f2_dup(q.x), qyh = f2_dup(q.y), qxl = f2_dup(q.z), qyl = f2_dup(q.w);
        const f2 k2h2 = f2_dup(k2h), k2l2 = f2_dup(k2l), cut2 = f2_dup(cutf);
        // part: the candidates of a bin row since the last multiple of kLooSum
        // of the group's range in it (a group's queries are all summed in the
        // same pieces), then into the compensated sum
        float s = 0.0f, c = 0.0f, part = 0.0f;
        auto flush = [&] {
            const float y = part - c;
            const float tt = s + y;
            c = (tt - s) - y;
            s = tt;
            part = 0.0f;
        };
        unsigned cnt = 0;
        // The item's bin rows, 32 at a time.  The candidates of a stretch of
        // rows are numbered through in slots, each row's from a multiple of
        // kLooTrip of the group's range and to a whole number of trips.
        for (int rb = by0; rb <= by1; rb += 32) {
            __syncwarp();  // the previous stretch's tables have been read
            {
                // a point of the row can be in reach of the box only within
                // sqrt(reach^2 - dy^2) of it, dy the rows' distance (a lower
                // bound): the window is the box grown by a disc
                int4 rw = make_int4(0, 0, 0, 0);
                const int by = rb + lane;
                if (by <= by1) {
                    const double rlo = L.oy + (double)by * L.side, rhi = rlo + L.side;
                    const double dy = fmax(0.0, fmax(rlo - (double)mxy, (double)mny - rhi)) * (1.0 - 1e-9);
                    const double rr = reach * reach - dy * dy;
                    if (rr >= 0.0) {
                        const double hw = sqrt(rr) * (1.0 + 1e-9) + 1e-9 * reach;
                        const double f0 = fmax(g0, floor(((double)mnx - hw - L.ox) * L.inv_side));
                        const double f1 = fmin(g1, floor(((double)mxx + hw - L.ox) * L.inv_side));
                        if (f0 <= f1) {
                            const int32_t* bs = L.bin_start + (int64_t)by * L.nbx;
                            rw.z = bs[(int64_t)g0];
                            rw.y = (bs[(int64_t)f0] - rw.z) / kLooTrip * kLooTrip;
                            rw.w = bs[(int64_t)f1 + 1] - rw.z;
                        }
                    }
                }
                const int len = rw.w > rw.y ? (rw.w - rw.y + kLooTrip - 1) / kLooTrip * kLooTrip : 0;
                int end = len;
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, end, o);
                    if (lane >= o) end += v;
                }
                rw.x = end;
                rw.y -= end - len;
                row[lane] = rw;
            }
            __syncwarp();
            // this part's slots, between multiples of kLooSum of the rows' ranges
            const int64_t T = row[31].x;
            auto part_at = [&](int sp) {
                int j = (int)(T * sp / P.nsplit), i = 0, pre = 0;
                if (sp == 0 || sp == P.nsplit || T == 0) return j;  // (no row ends beyond slot 0 if T is 0)
                while (j >= row[i].x) pre = row[i++].x;
                j = (j + row[i].y) / kLooSum * kLooSum - row[i].y;
                return max(j, pre);
            };
            const int j0 = part_at(split), j1 = part_at(split + 1);
            // the query's own slot
            const int jself =
                qv && qby >= rb && qby < rb + 32 ? qpos - row[qby - rb].z - row[qby - rb].y : -1;
            // the row of this lane's next candidate
            int r = 0, pre = 0;
            int4 rw = row[0];
            // this lane's two candidates of the coming batch
            float4 cp[2];
            float cw[2];
            unsigned new_sum[2];  // bit b: the trip that starts at the b-th slot begins a piece of its row
            auto fetch = [&](int jb) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int j = jb + 32 * i;
                    cp[i] = make_float4(INFINITY, 0.0f, 0.0f, 0.0f);  // past the end: beyond the cutoff of any h
                    cw[i] = 0.0f;
                    bool first = false;
                    int o = INT_MAX;
                    if (j < j1) {
                        while (j >= rw.x) {
                            pre = rw.x;
                            rw = row[++r];
                        }
                        o = j + rw.y;
                        first = j == pre || o % kLooSum == 0;
                    }
                    new_sum[i] = __ballot_sync(0xffffffffu, first);
                    if (o >= rw.w) continue;
                    const int cpos = rw.z + o;
                    cp[i] = *reinterpret_cast<const float4*>(pts + cpos);
                    if (wl) {
                        cw[i] = wl[cpos];
                    } else {
                        cw[i] = pts[cpos].wk;
                        if (P.ew) {
                            const int64_t pi = L.perm[cpos], ch = pi / P.ew_chunk;
                            cw[i] *= P.ew[(int64_t)k * P.ew_chunk + ch * P.ew_cstride + (pi - ch * P.ew_chunk)];
                        }
                    }
                }
            };
            auto put = [&](int buf) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    cand[buf][0][lane + 32 * i] = cp[i].x;
                    cand[buf][1][lane + 32 * i] = cp[i].y;
                    cand[buf][2][lane + 32 * i] = cp[i].z;
                    cand[buf][3][lane + 32 * i] = cp[i].w;
                    cand[buf][4][lane + 32 * i] = cw[i];
                }
            };
            int buf = 0;
            fetch(j0 + lane);
            put(0);
            __syncwarp();
            flush();
            for (int j = j0; j < j1; j += kLooB) {
                const int m = min(kLooB, j1 - j);
                const bool more = j + kLooB < j1;
                const unsigned long long pieces = ((unsigned long long)new_sum[1] << 32) | new_sum[0];
                if (more) fetch(j + kLooB + lane);
#pragma unroll 1
                for (int t = 0; t < m; t += kLooTrip) {
                    if ((pieces >> t) & 1u) flush();
                    // x < 0: inside the cutoff; the term is p times the weight ws
                    float p[kLooTrip], x[kLooTrip], ws[kLooTrip];
#pragma unroll
                    for (int u = 0; u < kLooTrip; u += 2) {
                        const f2 xh = *reinterpret_cast<const f2*>(&cand[buf][0][t + u]);
                        const f2 yh = *reinterpret_cast<const f2*>(&cand[buf][1][t + u]);
                        const f2 xl = *reinterpret_cast<const f2*>(&cand[buf][2][t + u]);
                        const f2 yl = *reinterpret_cast<const f2*>(&cand[buf][3][t + u]);
                        const f2 w = *reinterpret_cast<const f2*>(&cand[buf][4][t + u]);
                        const f2 dx = f2_add(f2_sub(xh, qxh), f2_sub(xl, qxl));
                        const f2 dy = f2_add(f2_sub(yh, qyh), f2_sub(yl, qyl));
                        const f2 d2 = f2_fma(dx, dx, f2_mul(dy, dy));
                        f2_get(f2_sub(d2, cut2), x[u], x[u + 1]);
                        // 2^-a = 2^-n 2^-g with a = n + g, |g| <= 1/2.  2^-n comes from the
                        // special-function unit, which is exact for integers and idle
                        // otherwise, not from a shift into the exponent bits
                        const f2 a = f2_fma(d2, k2h2, f2_mul(d2, k2l2));
                        const f2 n = f2_sub(f2_sub(magic, a), magic);  // -n
                        float g0, g1, n0, n1;
                        f2_get(f2_add(a, n), g0, g1);
                        f2_get(n, n0, n1);
                        p[u] = mgk_exp2_neg_frac(g0);
                        p[u + 1] = mgk_exp2_neg_frac(g1);
                        f2_get(f2_mul(w, f2_make(mgk_ex2(n0), mgk_ex2(n1))), ws[u], ws[u + 1]);
                    }
                    const int ts = jself - (j + t);  // the query's own place in the trip, if in it
                    float near = fabsf(x[0]);
#pragma unroll
                    for (int u = 1; u + 1 < kLooTrip; u += 2) near = mgk_min3(near, fabsf(x[u]), fabsf(x[u + 1]));
                    near = fminf(near, fabsf(x[kLooTrip - 1]));
                    if (near <= epsd2 || (unsigned)ts < (unsigned)kLooTrip) {
#pragma unroll
                        for (int u = 0; u < kLooTrip; u++) {
                            if (fabsf(x[u]) <= epsd2) {  // near the cutoff: the oracle's FP64 decision
                                int rr = 0;
                                while (j + t + u >= row[rr].x) rr++;
                                const float4 cc =
                                    *reinterpret_cast<const float4*>(pts + (j + t + u + row[rr].y + row[rr].z));
                                x[u] = mgk_d2_exact(qx, qy, cc.x + cc.z, cc.y + cc.w) < cut ? -1.0f : 1.0f;
                            }
                            if (u == ts) x[u] = 1.0f;  // the query itself
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kLooTrip; u++) {
                        if (x[u] < 0.0f) part = __fmaf_rn(p[u], ws[u], part);
                        cnt += __float_as_uint(x[u]) >> 31;
                    }
                }
                if (more) put(buf ^ 1);
                __syncwarp();  // this batch has been scanned, the next one is in place
                buf ^= 1;
            }
        }
        flush();
        if (qv) cnt_all += cnt;
        const double sum_q = (double)s - (double)c;
        if (P.psum) {
            P.psum[(((int64_t)split * P.nh + k) * ngs + gi) * 32 + lane] = sum_q;
        } else {
            const double sum = warp_sum(qv ? loo_log(sum_q, h2) : 0.0);
            if (lane == 0) P.part[(int64_t)k * ngs + gi] = sum;
        }
    }
    if (P.evals) {
        for (int o = 16; o; o >>= 1) cnt_all += __shfl_xor_sync(0xffffffffu, cnt_all, o);
        if (lane == 0 && cnt_all) atomicAdd(P.evals, cnt_all);
    }
}

// The log sums of the groups' quarters from the parts' sums of each query,
// added in order (one warp per quarter).
__global__ void __launch_bounds__(kLooWarps * 32) k_loo_combine(LooParams P) {
    const int lane = threadIdx.x & 31, gi = blockIdx.x * kLooWarps + (threadIdx.x >> 5);
    const int64_t ngs = (int64_t)P.gcount * kLooSub;
    if (gi >= ngs) return;
    for (int k = blockIdx.y; k < P.nh; k += gridDim.y) {
        double lg = 0.0;
        if ((int64_t)P.g0 * kLooQ + (int64_t)gi * 32 + lane < P.n) {
            double v = 0.0;
            for (int sp = 0; sp < P.nsplit; sp++) v += P.psum[(((int64_t)sp * P.nh + k) * ngs + gi) * 32 + lane];
            lg = loo_log(v, mgk_h2(P.hgrid[k]));
        }
        const double sum = warp_sum(lg);
        if (lane == 0) P.part[k * ngs + gi] = sum;
    }
}

// logL[k] = fixed-order sum of the group partials of h_k (one CTA per h).  The
// last CTA to finish takes the first index of the largest (ties resolve to the
// lower index; a NaN is never larger, nor anything than one at index 0).
__global__ void __launch_bounds__(256) k_loo_finish(LooParams P, LooHost H, int ngroups, double* __restrict__ logl) {
    __shared__ double sh[256];
    __shared__ bool last;
    const int k = blockIdx.x;
    double v = 0.0;
    for (int i = threadIdx.x; i < ngroups; i += blockDim.x) v += P.part[(int64_t)k * ngroups + i];
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        logl[k] = sh[0];
        H.logl[k] = sh[0];
        __threadfence();
        last = atomicAdd(&P.counter[1], 1u) == (unsigned)P.nh - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x >= 32) return;
    __threadfence();
    const volatile double* l = logl;
    const int lane = threadIdx.x;
    double top = l[0];
    int best = 0;
    for (int i = lane; i < P.nh; i += 32) {
        const double w = l[i];
        if (w > top) {
            top = w;
            best = i;
        }
    }
    for (int o = 16; o; o >>= 1) {
        const double w = __shfl_xor_sync(0xffffffffu, top, o);
        const int b = __shfl_xor_sync(0xffffffffu, best, o);
        if (w > top || (w == top && b < best)) {
            top = w;
            best = b;
        }
    }
    if (lane == 0) *H.best = best;
    if (lane < 2) H.evals[lane] = P.evals[lane - 1];
}

}  // namespace

// ---- the batch object ------------------------------------------------------
struct mgk_loo_batch {
    mgk_ctx* ctx = nullptr;
    const mgk_points* pts = nullptr;
    const mgk_raster* mask = nullptr;
    int64_t n = 0;
    int nh = 0;
    int ngroups = 0;
    int g0 = 0, gcount = 0;  // the share's query groups
    std::vector<mgk_index*> lev;
    std::vector<int32_t*> qord;  // per level
    float* d_h = nullptr;
    float* d_ew = nullptr;
    LevelDesc* d_lev = nullptr;
    cudaStream_t cap = nullptr;  // capture stream
    int* d_korder = nullptr;
    int* d_klevel = nullptr;
    float* d_wl = nullptr;
    double* d_psum = nullptr;
    double* d_part = nullptr;
    double* d_logl = nullptr;
    unsigned* d_counter = nullptr;
    unsigned long long* d_evals = nullptr;  // [0] edge, [1] loo
    char* h_io = nullptr;  // the run's numbers (LooHost) at the host's address
    LooHost io{};
    size_t o_logl = 0, o_evals = 0, o_best = 0;  // offsets in h_io (the bandwidths come first)
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    LooParams P{};
    size_t bytes_ew = 0, bytes_wl = 0, bytes_psum = 0, bytes_part = 0;
    int grid = 1;
};

// Bandwidths that one launch of the scan takes: all but for very long lists of very many points.
static int scan_part(const mgk_loo_batch* B) {
    const int64_t per_h = (int64_t)B->P.gcount * kLooSub * B->P.nsplit;
    return (int)std::min<int64_t>(B->nh, std::max<int64_t>(1, kMaxItems / std::max<int64_t>(per_h, 1)));
}

// Kernels of a batch, the edge weights' aside.
static int loo_launches(const mgk_loo_batch* B) {
    const int scans = (B->nh + scan_part(B) - 1) / scan_part(B);
    return 2 + (B->P.wl ? 1 : 0) + (B->P.gcount > 0 ? scans : 0) + (B->P.gcount > 0 && B->P.psum ? 1 : 0);
}

static int loo_enqueue(mgk_loo_batch* B) {
    mgk_ctx* ctx = B->ctx;
    cudaStream_t s = ctx->stream;
    k_loo_prep<<<1, 256, 0, s>>>(B->P, B->io, B->d_h, B->d_lev);
    if (B->mask) {
        int st = mgk_launch_edge_weights_multi(ctx, B->n, B->pts->x, B->pts->y, nullptr, 0.0f, B->d_h, B->nh,
                                               B->pts->dist2, B->mask, B->d_ew, B->n, B->d_evals);
        if (st) return st;
    }
    if (B->P.wl) {
        const unsigned gx = (unsigned)std::min<int64_t>((B->n + 255) / 256, 4 * (int64_t)ctx->sm_count);
        k_loo_weights<<<dim3(gx, std::min((unsigned)B->nh, kMaxGridY)), 256, 0, s>>>(B->P);
    }
    if (B->P.gcount > 0) {
        LooParams P = B->P;
        for (P.k0 = 0; P.k0 < B->nh; P.k0 = P.k1) {
            P.k1 = P.k0 + std::min(scan_part(B), B->nh - P.k0);
            if (P.k0) MGK_CHECK_CUDA(ctx, cudaMemsetAsync(B->d_counter, 0, sizeof(unsigned), s));
            k_loo_multi<<<(unsigned)B->grid, kLooWarps * 32, 0, s>>>(P);
        }
        if (B->P.psum)
            k_loo_combine<<<dim3((unsigned)((B->P.gcount * kLooSub + kLooWarps - 1) / kLooWarps),
                                 std::min((unsigned)B->nh, kMaxGridY)),
                            kLooWarps * 32, 0, s>>>(B->P);
    }
    k_loo_finish<<<B->nh, 256, 0, s>>>(B->P, B->io, B->P.gcount * kLooSub, B->d_logl);
    MGK_CHECK_LAUNCH(ctx, "loo batch");
    MGK_COUNT_LAUNCH(ctx, loo_launches(B));
    return MGK_OK;
}

void mgk_loo_batch_destroy(mgk_loo_batch* B) {
    if (!B) return;
    mgk_ctx* c = B->ctx;
    if (B->exec) cudaGraphExecDestroy(B->exec);
    if (B->graph) cudaGraphDestroy(B->graph);
    if (B->cap) cudaStreamDestroy(B->cap);
    mgk_free(c, B->d_lev, sizeof(LevelDesc) * kMaxLev);
    for (int32_t* q : B->qord) mgk_free(c, q, sizeof(int32_t) * (size_t)std::max<int64_t>(B->n, 1));
    for (mgk_index* i : B->lev) mgk_index_destroy(i);
    const size_t nh = (size_t)B->nh;
    mgk_free(c, B->d_h, sizeof(float) * nh);
    mgk_free(c, B->d_ew, B->bytes_ew);
    mgk_free(c, B->d_korder, sizeof(int) * nh);
    mgk_free(c, B->d_klevel, sizeof(int) * nh);
    mgk_free(c, B->d_wl, B->bytes_wl);
    mgk_free(c, B->d_psum, B->bytes_psum);
    mgk_free(c, B->d_part, B->bytes_part);
    mgk_free(c, B->d_logl, sizeof(double) * nh);
    mgk_free(c, B->d_counter, 2 * sizeof(unsigned));
    mgk_free(c, B->d_evals, 2 * sizeof(unsigned long long));
    delete B;
}

// Plans a batch of nh bandwidths within [h_lo, h_hi]: one point index per
// bandwidth octave, buffers, and the captured graph.
int mgk_loo_batch_create(mgk_ctx* c, const mgk_points* p, const mgk_raster* r, float h_lo, float h_hi, int nh,
                         mgk_loo_batch** out) {
    return mgk_loo_batch_create_share(c, p, r, h_lo, h_hi, nh, 0, 1, nullptr, 0, out, true);
}

// Share `part` of `nparts` of a batch: the query groups
// [part G / nparts, (part + 1) G / nparts) of every h, G = ceil(n / 128).
// ew_ext (device, optional, with r == NULL): the edge weights of every point
// and h in chunks of ew_chunk points, each nh rows of ew_chunk floats.
int mgk_loo_batch_create_share(mgk_ctx* c, const mgk_points* p, const mgk_raster* r, float h_lo, float h_hi,
                               int nh, int part, int nparts, const float* ew_ext, int64_t ew_chunk,
                               mgk_loo_batch** out, bool replay) {
    mgk_loo_batch* B = new (std::nothrow) mgk_loo_batch();
    if (!B) return mgk_fail(c, MGK_ERR_INVALID, "loo batch: out of host memory");
    B->ctx = c;
    B->pts = p;
    B->mask = r;
    B->n = p->n;
    B->nh = nh;
    B->ngroups = (int)((p->n + kLooQ - 1) / kLooQ);
    B->g0 = (int)((int64_t)B->ngroups * part / nparts);
    B->gcount = (int)((int64_t)B->ngroups * (part + 1) / nparts) - B->g0;
    int st = MGK_OK;
    // levels: bin sides 0.75 h_lo * 2^l up to the side for h_hi
    mgk_points view = *p;  // index over w only; e(h) is applied per h
    view.has_ew = false;
    view.h = nullptr;
    const int nlev = std::min(kMaxLev, 1 + std::max(0, (int)std::ceil(std::log2((double)h_hi / (double)h_lo))));
    mgk_extent ext;
    st = mgk_points_extent(c, &view, false, &ext);
    if (st == MGK_OK) st = mgk_index_build_levels(c, &view, h_lo, 0.75 * (double)h_lo, nlev, &ext, &B->lev, &B->qord);
    const size_t n1 = (size_t)std::max<int64_t>(p->n, 1);
    B->bytes_ew = r ? sizeof(float) * n1 * (size_t)nh : 16;
    B->bytes_part = sizeof(double) * (size_t)nh * (size_t)std::max(B->gcount, 1) * kLooSub;
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_h, sizeof(float) * nh);
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_ew, B->bytes_ew);
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_korder, sizeof(int) * nh);
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_klevel, sizeof(int) * nh);
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_part, B->bytes_part);
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_logl, sizeof(double) * nh);
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_counter, 2 * sizeof(unsigned));
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_evals, 2 * sizeof(unsigned long long));
    if (st == MGK_OK) st = mgk_alloc(c, (void**)&B->d_lev, sizeof(LevelDesc) * kMaxLev);
    // Parts of a group's candidates: enough work items for about four rounds of
    // the resident warps (a golden-section step on 20,000 points has 1,256 items
    // for 2,368 warps, the dense groups' the longest: 3.33 ms per search with
    // four rounds, 3.41 with three, 3.57 with two, 4.12 with one), for two below
    // 2^13 points, whose items are short (16 bandwidths on 2,000 points 281 us
    // with two, 283 with four; 8,000 points the same with both).  From the whole
    // problem's groups, so a share of it sums each query as the whole does.
    int nsplit = 1;
    int occ = 1;
    if (st == MGK_OK && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_loo_multi, kLooWarps * 32, 0) != cudaSuccess)
        st = mgk_fail(c, MGK_ERR_CUDA, "loo batch: occupancy");
    const int64_t resident = (int64_t)c->sm_count * std::max(occ, 1) * kLooWarps;  // warps
    const int64_t items = (int64_t)nh * std::max(B->ngroups, 1) * kLooSub;
    const int64_t want = (p->n < (1 << 13) ? 2 : 4) * resident;
    if (items < want) nsplit = (int)std::min<int64_t>(kMaxSplit, (want + items - 1) / items);
    // What follows is left out where there is no memory for it, so it comes after
    // all that is needed: the runs, and for one bandwidth the blocks that the edge
    // weights take during the run (held here, and in the pool by then).
    if (st == MGK_OK && r) st = mgk_raster_runs(c, const_cast<mgk_raster*>(r));
    const size_t b_later[2] = {sizeof(int) * n1, 2 * sizeof(int)};
    void* later[2] = {};
    if (r && nh == 1)
        for (int i = 0; i < 2 && st == MGK_OK; i++) st = mgk_alloc(c, &later[i], b_later[i]);
    if (st == MGK_OK && nsplit > 1) {
        B->bytes_psum = sizeof(double) * (size_t)nsplit * (size_t)nh * (size_t)std::max(B->gcount, 1) * kLooQ;
        if (mgk_alloc(c, (void**)&B->d_psum, B->bytes_psum)) nsplit = 1;  // no memory: whole groups
    }
    // The weights in record order are a shortcut: without the memory for them
    // the scan gathers each weight through the permutation.
    const bool has_ew = r || ew_ext;
    if (st == MGK_OK && has_ew && p->n > 0) {
        B->bytes_wl = sizeof(float) * n1 * (size_t)nh;
        if (mgk_alloc(c, (void**)&B->d_wl, B->bytes_wl)) B->d_wl = nullptr;
    }
    for (int i = 0; i < 2; i++) mgk_free(c, later[i], b_later[i]);
    // a staging slot of the context (a batch lives within one call, whose
    // extent above has waited for the slot's former users)
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    const size_t o_lev = up(sizeof(float) * nh);
    B->o_logl = o_lev + up(sizeof(LevelDesc) * kMaxLev);
    B->o_evals = B->o_logl + up(sizeof(double) * nh);
    B->o_best = B->o_evals + 2 * sizeof(unsigned long long);
    char* d_io = nullptr;
    if (st == MGK_OK) st = mgk_host_stage_slot(c, 2, B->o_best + 256, (void**)&B->h_io, (void**)&d_io);
    if (st == MGK_OK && p->n == 0 && cudaStreamSynchronize(c->stream) != cudaSuccess)
        st = mgk_fail(c, MGK_ERR_CUDA, "loo batch: stream");
    if (st) {
        mgk_loo_batch_destroy(B);
        return st;
    }
    LooParams& P = B->P;
    P.nlev = (int)B->lev.size();
    LevelDesc* hl = reinterpret_cast<LevelDesc*>(B->h_io + o_lev);
    for (int l = 0; l < P.nlev; l++) {
        const mgk_index* I = B->lev[l];
        hl[l] = LevelDesc{I->pts, I->bin_start, I->perm, B->qord[l], I->ox, I->oy, I->side, 1.0 / I->side, I->nbx,
                          I->nby};
        P.side[l] = I->side;
    }
    B->io = LooHost{(const float*)d_io, (const LevelDesc*)(d_io + o_lev), (double*)(d_io + B->o_logl),
                    (unsigned long long*)(d_io + B->o_evals), (int*)(d_io + B->o_best)};
    P.lev = B->d_lev;
    P.n = p->n;
    P.g0 = B->g0;
    P.gcount = B->gcount;
    P.nh = nh;
    P.hgrid = B->d_h;
    P.korder = B->d_korder;
    P.klevel = B->d_klevel;
    if (r) {
        P.ew = B->d_ew;
        P.ew_chunk = std::max<int64_t>(p->n, 1);
    } else if (ew_ext) {
        P.ew = ew_ext;
        P.ew_chunk = std::max<int64_t>(ew_chunk, 1);
    } else {
        P.ew = nullptr;
        P.ew_chunk = 1;
    }
    P.ew_cstride = P.ew_chunk * (int64_t)nh;
    P.nsplit = nsplit;
    P.wl = B->d_wl;
    P.psum = nsplit > 1 ? B->d_psum : nullptr;
    P.part = B->d_part;
    B->grid = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)nh * B->gcount * kLooSub * nsplit + kLooWarps - 1) / kLooWarps,
                                                     resident / kLooWarps));
    P.counter = B->d_counter;
    P.evals = B->d_evals + 1;
    // capture the sequence into a graph on a private stream (the graph is
    // then launched into the context's stream); if capture fails, or the
    // batch runs once (replay false: capture and instantiation would cost
    // more than they save), the batch launches its kernels directly
    if (replay && cudaStreamSynchronize(c->stream) == cudaSuccess &&
        cudaStreamCreateWithFlags(&B->cap, cudaStreamNonBlocking) == cudaSuccess &&
        cudaStreamBeginCapture(B->cap, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        cudaStream_t keep = c->stream;
        const uint64_t l0 = c->launches;
        c->stream = B->cap;
        const int est = loo_enqueue(B);
        c->stream = keep;
        c->launches = l0;  // counted at each replay
        cudaGraph_t g = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(B->cap, &g);
        if (est == MGK_OK && ce == cudaSuccess && g) {
            B->graph = g;
            if (cudaGraphInstantiate(&B->exec, g, 0) != cudaSuccess) B->exec = nullptr;
        } else if (g) {
            cudaGraphDestroy(g);
        }
        cudaGetLastError();
    }
    *out = B;
    return MGK_OK;
}

// Scores the nh bandwidths hs (host) of a planned batch: logL, argmax and the
// edge and LOO eval counts.
int mgk_loo_batch_run(mgk_loo_batch* B, const float* hs, double* logl, int* best, int64_t* edge_evals,
                      int64_t* loo_evals) {
    mgk_ctx* c = B->ctx;
    cudaStream_t s = c->stream;
    memcpy(B->h_io, hs, sizeof(float) * (size_t)B->nh);
    MGK_CHECK_CUDA(c, cudaEventRecord(c->ev_a, s));
    if (B->exec) {
        MGK_CHECK_CUDA(c, cudaGraphLaunch(B->exec, s));
        MGK_COUNT_LAUNCH(c, loo_launches(B) + (B->mask ? 1 : 0));
    } else {
        int st = loo_enqueue(B);
        if (st) return st;
    }
    MGK_CHECK_CUDA(c, cudaEventRecord(c->ev_b, s));
    MGK_CHECK_CUDA(c, cudaStreamSynchronize(s));
    memcpy(logl, B->h_io + B->o_logl, sizeof(double) * (size_t)B->nh);
    const unsigned long long* tail = reinterpret_cast<const unsigned long long*>(B->h_io + B->o_evals);
    const int* hb = reinterpret_cast<const int*>(B->h_io + B->o_best);
    if (best) *best = *hb;
    if (edge_evals) *edge_evals = (int64_t)tail[0];
    if (loo_evals) *loo_evals = (int64_t)tail[1];
    c->last_loo_evals[0] = (int64_t)tail[0];
    c->last_loo_evals[1] = (int64_t)tail[1];
    cudaEventElapsedTime(&c->last_loo_ms, c->ev_a, c->ev_b);
    return MGK_OK;
}
