// Adaptive bandwidths (h_option 2): Hooke-Jeeves search over (h0, alpha).
//
// The reference (main, kde_cuda_kdtr_tiled.cu:548-573) starts from the
// rule-of-thumb h0 with alpha0 = -0.5 and searches (hooke_jeeves /
// hj_likelihood, :3677-3785) for the (h, alpha) maximising
// LogLikelihood(h, alpha) (CPU branch :3553-3650):
//   1. edge weights e(h) at the fixed h,
//   2. pilot density at every point, itself included:
//        den0_j = sum_{i, d^2 < 9h^2} K_h(d) w_i e_i(h),
//   3. hs_i = h (den0_i / gml)^alpha, gml the geometric mean of den0 (compGML),
//   4. edge weights e(hs) at the per-point bandwidths,
//   5. leave-one-out density with the bandwidth of each source point:
//        den1_j = sum_{i != j, d^2 < 9 hs_i^2} K_{hs_i}(d) w_i e_i(hs),
//   6. logL = sum_j log max(den1_j, EPSILONDENSITY).
// After the search the bandwidths of the optimum are computed once more
// (steps 1-3) and used for the density raster.
//
// On the device: steps 1 and 4 are k_edge_rows; steps 2 and 5 are
// k_point_density over a cell-binned index of the points (fixed-h index for
// the pilot, per-point-h index for the LOO sum), one lane per query, the
// candidates staged through shared memory, the cutoff decided in FP32 with a
// band re-decided by the oracle's FP64 test, terms from an unbiased
// polynomial exp2, Kahan-compensated FP32 partials and an FP64 result per
// point; the geometric mean, the bandwidths and the log sum are FP64 on the
// device (fixed-order reductions).  The search itself runs on the host with
// the reference's float step arithmetic and its bookkeeping of the five
// likelihoods.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>

#include "mgk_internal.cuh"

namespace {

constexpr int kPdQ = 32;    // queries of a CTA, one per lane of its one warp
constexpr int kPdB = 64;    // candidates per staged batch, two per lane
constexpr int kPdTrip = 8;  // candidates scanned at a time
// Candidates summed in plain FP32 before each Kahan step.  The sums' own error,
// FP32 emulated on 18,000 clustered points with per-point h: 4.6e-8 rms (1.6e-7
// at most) with the whole batch of 64, 3.2e-8 (0.9e-7) with 32, 1.9e-8 (0.6e-7)
// with 16; pieces of 32 ended by every bin row, 2.9e-8 (1.2e-7).
constexpr int kPdSum = 16;
static_assert(kPdB % kPdSum == 0 && kPdSum % kPdTrip == 0, "whole pieces of whole trips");
constexpr int kPdSeg = 64;  // runs of bins scanned together
// Warps per SM to split a launch into: fourteen rounds of the 16 that are
// resident (groups in clusters take longest and leave slots idle in the tail; a
// search on 50,000 points takes 22.6 ms with six rounds, 22.9 with nine, 22.5
// with fourteen, smaller ones the same with each)
constexpr int kPdWarps = 224;
// Points from which the queries go along a curve: making the order takes 90 us
// of a search (records' order / curve: 400 points 2.96 / 3.05 ms, 5,000 5.47 /
// 5.52, 10,000 5.95 / 5.74, 50,000 24.1 / 22.8)
constexpr int64_t kPdCurve = 1 << 13;
// The cutoff of per-point h in exponents, 9 h^2 log2(e) / (2 h^2) for every h,
// and the relative band around a cutoff in which FP32 does not decide.
constexpr float kPdCut = (float)(0.5 * MGK_CUT * MGK_LOG2E);
constexpr float kPdBand = 4e-6f;

// psum[y][q] = sum over candidates i (the points of the index within reach
// of the CTA's 32 queries, in the bin rows y, y + nsplit, ... of
// the window, y = blockIdx.y) of [in cutoff] K w_i e_i, unnormalised.  Fixed h
// (the pilot density): the query itself included, terms exp2(-d^2 k2) w e;
// per-point h (VARH, the leave-one-out density): without the query itself, the
// candidate's own k2 and cutoff, weights already carry 1/(h_i^2 TWO_PI).
// Splitting the rows over nsplit CTAs gives a
// launch enough CTAs for the whole GPU when there are few queries.
//
// The queries are the points along a Hilbert curve (order; record inv[order[q]]),
// so that the box around 32 of them is small in both directions: 13 % fewer
// candidates than the records' order (stretches of bin rows, and whole rows
// where a group passes from one to the next) on 50,000 clustered points, where
// a search takes 22.9 ms instead of 24.1, and a third of them on uniform
// points.  Few points, or no memory for the order: the records' order.
//
// The candidates are runs of bins: with fixed h one run per bin row (the box
// around the queries grown by a disc), with per-point h the bins of the row
// whose own largest reach (bin_r2: 9 h^2 of its widest point) can touch the
// box, so points with small h far from the group are not tested even where a
// wide point lies beyond them.  Up to 64 runs are numbered through and scanned
// as one list, two candidates at a time in packed FP32 (f32x2).
//
// Bound by the issue slots and the FMA pipe, as the leave-one-out scan is
// (about 25 instructions per candidate and warp).  50,000 points, one
// likelihood's sum with per-point h: 1.06 ms with 128 queries a CTA, scalar
// FP32 and one span of bins per row, 0.41 ms now.
template <bool VARH>
__global__ void __launch_bounds__(kPdQ, 16) k_point_density(int64_t n, const MgkPt* __restrict__ pts,
                                                            const int32_t* __restrict__ bin_start, double ox,
                                                            double oy, double side, int64_t nbx, int64_t nby,
                                                            double reach, double h2, const float* __restrict__ bin_r2,
                                                            const int32_t* __restrict__ order,
                                                            const int32_t* __restrict__ inv,
                                                            double* __restrict__ psum,
                                                            unsigned long long* __restrict__ evals) {
    // candidates by component: xh, yh, xl, yl, weight, k2h, k2l; two batches
    constexpr int kComp = VARH ? 7 : 5;
    __shared__ __align__(16) float cand[2][kComp][kPdB];
    __shared__ int2 seg[kPdSeg];  // slots before its end, what takes a slot to its record
    const double inv_side = 1.0 / side;
    int lane;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));  // kept in a register
    const unsigned lt = (1u << lane) - 1u;
    const int64_t slot = (int64_t)blockIdx.x * kPdQ + lane;
    const bool qv = slot < n;
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int64_t qpos = slot;
    if (qv && order) qpos = inv[order[slot]];
    if (qv) q = *reinterpret_cast<const float4*>(pts + qpos);
    const float qx = q.x + q.z, qy = q.y + q.w;
    float mnx = qv ? qx : FLT_MAX, mxx = qv ? qx : -FLT_MAX, mny = qv ? qy : FLT_MAX, mxy = qv ? qy : -FLT_MAX;
    for (int o = 16; o; o >>= 1) {
        mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
        mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
        mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
        mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
    }
    const int by0 = (int)fmax(0.0, floor(((double)mny - reach - oy) * inv_side));
    const int by1 = (int)fmin((double)(nby - 1), floor(((double)mxy + reach - oy) * inv_side));
    // fixed-h constants
    const double k2 = MGK_LOG2E / (2.0 * h2);
    const f2 k2hc = f2_dup((float)k2), k2lc = f2_dup((float)(k2 - (double)(float)k2));
    const f2 qxh = f2_dup(q.x), qyh = f2_dup(q.y), qxl = f2_dup(q.z), qyl = f2_dup(q.w);
    // fixed h: the cutoff of d^2 itself
    const float cutf = VARH ? kPdCut : (float)(MGK_CUT * h2), band = kPdBand * cutf;
    const f2 cut2 = f2_dup(cutf), magic = f2_dup(12582912.0f);
    // past the end: beyond every cutoff, for any h (with fixed h the exponent of
    // a finite distance may overflow to either side)
    constexpr float kFar = VARH ? 1e18f : INFINITY;
    float s = 0.0f, c = 0.0f, part = 0.0f;
    auto flush = [&] {
        const float y = part - c;
        const float tt = s + y;
        c = (tt - s) - y;
        s = tt;
        part = 0.0f;
    };
    unsigned cnt = 0;
    int nseg = 0;
    // Scans the nseg runs in seg, there as (candidates, first record).
    auto scan = [&] {
        __syncwarp();
        const int2 e0 = lane < nseg ? seg[lane] : make_int2(0, 0);
        const int2 e1 = lane + 32 < nseg ? seg[lane + 32] : make_int2(0, 0);
        int p0 = e0.x, p1 = e1.x;
        for (int o = 1; o < 32; o <<= 1) {
            const int v0 = __shfl_up_sync(0xffffffffu, p0, o), v1 = __shfl_up_sync(0xffffffffu, p1, o);
            if (lane >= o) {
                p0 += v0;
                p1 += v1;
            }
        }
        p1 += __shfl_sync(0xffffffffu, p0, 31);
        const int T = __shfl_sync(0xffffffffu, p1, 31);
        seg[lane] = make_int2(p0, e0.y - (p0 - e0.x));
        seg[lane + 32] = make_int2(p1, e1.y - (p1 - e1.x));
        __syncwarp();
        // the query's own slot
        int jself = -1;
        if (VARH) {
            int pre = 0;
            for (int i = 0; i < nseg; i++) {
                const int2 g = seg[i];
                const int64_t j = qpos - g.y;
                if (j >= pre && j < g.x) jself = (int)j;
                pre = g.x;
            }
        }
        int r = 0;
        int2 sg = seg[0];
        float4 cp[2], cq[2];
        auto fetch = [&](int jb) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int j = jb + 32 * i;
                cp[i] = make_float4(kFar, 0.0f, 0.0f, 0.0f);
                cq[i] = make_float4(0.0f, 1.0f, 0.0f, 0.0f);
                if (j >= T) continue;
                while (j >= sg.x) sg = seg[++r];
                const float4* rec = reinterpret_cast<const float4*>(pts + (j + sg.y));
                cp[i] = rec[0];
                cq[i] = rec[1];  // wk, k2h, k2l, hh
            }
        };
        auto put = [&](int buf) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                cand[buf][0][lane + 32 * i] = cp[i].x;
                cand[buf][1][lane + 32 * i] = cp[i].y;
                cand[buf][2][lane + 32 * i] = cp[i].z;
                cand[buf][3][lane + 32 * i] = cp[i].w;
                cand[buf][4][lane + 32 * i] = cq[i].x;
                if (VARH) {
                    cand[buf][kComp - 2][lane + 32 * i] = cq[i].y;
                    cand[buf][kComp - 1][lane + 32 * i] = cq[i].z;
                }
            }
        };
        int buf = 0;
        fetch(lane);
        put(0);
        __syncwarp();
        for (int j = 0; j < T; j += kPdB) {
            const int m = min(kPdB, T - j);
            const bool more = j + kPdB < T;
            if (more) fetch(j + kPdB + lane);
#pragma unroll 1
            for (int t = 0; t < m; t += kPdTrip) {
                if (t % kPdSum == 0) flush();
                // x < 0: inside the cutoff; the term is p times the weight ws
                float p[kPdTrip], x[kPdTrip], ws[kPdTrip];
#pragma unroll
                for (int u = 0; u < kPdTrip; u += 2) {
                    auto at = [&](int k) { return *reinterpret_cast<const f2*>(&cand[buf][k][t + u]); };
                    const f2 dx = f2_add(f2_sub(at(0), qxh), f2_sub(at(2), qxl));
                    const f2 dy = f2_add(f2_sub(at(1), qyh), f2_sub(at(3), qyl));
                    const f2 d2 = f2_fma(dx, dx, f2_mul(dy, dy));
                    const f2 a = f2_fma(d2, VARH ? at(kComp - 2) : k2hc, f2_mul(d2, VARH ? at(kComp - 1) : k2lc));
                    f2_get(f2_sub(VARH ? a : d2, cut2), x[u], x[u + 1]);
                    const f2 m1 = f2_sub(f2_sub(magic, a), magic);  // -n, a = n + g
                    float g0, g1, n0, n1;
                    f2_get(f2_add(a, m1), g0, g1);
                    f2_get(m1, n0, n1);
                    p[u] = mgk_exp2_neg_frac(g0);
                    p[u + 1] = mgk_exp2_neg_frac(g1);
                    f2_get(f2_mul(at(4), f2_make(mgk_ex2(n0), mgk_ex2(n1))), ws[u], ws[u + 1]);
                }
                const int ts = jself - (j + t);  // the query's own place in the trip, if in it
                float near = fabsf(x[0]);
#pragma unroll
                for (int u = 1; u + 1 < kPdTrip; u += 2) near = mgk_min3(near, fabsf(x[u]), fabsf(x[u + 1]));
                near = fminf(near, fabsf(x[kPdTrip - 1]));
                if (near <= band || (unsigned)ts < (unsigned)kPdTrip) {
#pragma unroll
                    for (int u = 0; u < kPdTrip; u++) {
                        if (fabsf(x[u]) <= band) {  // near the cutoff: the oracle's FP64 decision
                            int i = 0;
                            while (j + t + u >= seg[i].x) i++;
                            const MgkPt cc = pts[j + t + u + seg[i].y];
                            const double cut = MGK_CUT * (VARH ? (double)cc.hh : h2);
                            x[u] = mgk_d2_exact(qx, qy, cc.xh + cc.xl, cc.yh + cc.yl) < cut ? -1.0f : 1.0f;
                        }
                        if (u == ts) x[u] = 1.0f;  // the query itself
                    }
                }
#pragma unroll
                for (int u = 0; u < kPdTrip; u++) {
                    if (x[u] < 0.0f) part = __fmaf_rn(p[u], ws[u], part);
                    cnt += __float_as_uint(x[u]) >> 31;
                }
            }
            if (more) put(buf ^ 1);
            __syncwarp();  // this batch has been scanned, the next one is in place
            buf ^= 1;
        }
        nseg = 0;
    };
    for (int by = by0 + (int)blockIdx.y; by <= by1; by += (int)gridDim.y) {
        // a point of the row can be in reach of the box only within
        // sqrt(reach^2 - dy^2) of it, dy the rows' distance (a lower bound)
        const double rlo = oy + (double)by * side, rhi = rlo + side;
        const double ddy = fmax(0.0, fmax(rlo - (double)mxy, (double)mny - rhi)) * (1.0 - 1e-9);
        const double rr = reach * reach - ddy * ddy;
        if (!(rr >= 0.0)) continue;
        const double hw = sqrt(rr) * (1.0 + 1e-9) + 1e-9 * reach;
        const double f0 = fmax(0.0, floor(((double)mnx - hw - ox) * inv_side));
        const double f1 = fmin((double)(nbx - 1), floor(((double)mxx + hw - ox) * inv_side));
        if (!(f0 <= f1)) continue;
        const int b0 = (int)f0, b1 = (int)f1;
        const int32_t* bs = bin_start + (int64_t)by * nbx;
        if constexpr (!VARH) {
            const int pos = bs[b0], len = bs[b1 + 1] - pos;
            if (len == 0) continue;
            if (nseg == kPdSeg) scan();
            if (lane == 0) seg[nseg] = make_int2(len, pos);
            nseg++;
        } else {
            for (int bx = b0; bx <= b1; bx += 32) {
                bool ok = false;
                int pos = 0, end = 0;
                if (bx + lane <= b1) {
                    const float r2 = bin_r2[(int64_t)by * nbx + bx + lane];
                    const double rx0 = ox + (double)(bx + lane) * side, rx1 = rx0 + side;
                    const double ddx = fmax(0.0, fmax(rx0 - (double)mxx, (double)mnx - rx1));
                    // a margin over the bin edges' rounding and the float h^2; r2 < 0: an empty bin
                    ok = r2 >= 0.0f && ddx * ddx + ddy * ddy <= (double)r2 * (1.0 + 1e-5) + 1e-6 * side * side;
                    if (ok) {
                        pos = bs[bx + lane];
                        end = bs[bx + lane + 1];
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, ok);
                const unsigned first = m & ~(m << 1);  // the lanes whose bin begins a run
                const int nrun = __popc(first);
                if (nseg + nrun > kPdSeg) scan();
                // the run's last bin: before the first clear bit above the lane's
                const unsigned gap = ~(m >> lane);
                const int last = gap ? lane + __ffs(gap) - 2 : 31;
                end = __shfl_sync(0xffffffffu, end, last & 31);
                if ((first >> lane) & 1u) seg[nseg + __popc(first & lt)] = make_int2(end - pos, pos);
                nseg += nrun;
            }
        }
    }
    if (nseg) scan();
    flush();
    if (qv) psum[(int64_t)blockIdx.y * n + slot] = (double)s - (double)c;
    if (evals) {
        if (!qv) cnt = 0;
        for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0 && cnt) atomicAdd(evals, (unsigned long long)cnt);
    }
}

constexpr int kPdC = 128;  // threads of the combining kernel

// den[order[q]] = the nsplit partials of query q summed in order (times
// 1/(h^2 TWO_PI) for a fixed h), and part[CTA] = the CTA's fixed-order sum of
// log(max(den, floor_v)).
__global__ void __launch_bounds__(kPdC) k_pd_combine(int64_t n, int nsplit, const double* __restrict__ psum,
                                                     const int32_t* __restrict__ order, bool varh, double h2,
                                                     double floor_v, double* __restrict__ den,
                                                     double* __restrict__ part) {
    __shared__ double s_lg[kPdC / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t q = (int64_t)blockIdx.x * kPdC + tid;
    double lg = 0.0;
    if (q < n) {
        double v = 0.0;
        for (int y = 0; y < nsplit; y++) v += psum[(int64_t)y * n + q];
        if (!varh) v /= h2 * (double)MGK_TWO_PI_F;
        den[order[q]] = v;
        lg = log(v > floor_v ? v : floor_v);
    }
    for (int o = 16; o; o >>= 1) lg += __shfl_xor_sync(0xffffffffu, lg, o);
    if (lane == 0) s_lg[warp] = lg;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int i = 0; i < kPdC / 32; i++) t += s_lg[i];
        part[blockIdx.x] = t;
    }
}

// out[0] = sum of the per-CTA partials in a fixed order (one CTA).
__global__ void k_sum_parts(int64_t g, const double* __restrict__ part, double* __restrict__ out) {
    __shared__ double sh[256];
    double a = 0.0;
    for (int64_t i = threadIdx.x; i < g; i += blockDim.x) a += part[i];
    sh[threadIdx.x] = a;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = sh[0];
}

// hs_i = h (den0_i / gml)^alpha with gml = exp(logsum / n), and the CTAs'
// largest of them (ordered bits, mapped host memory).  The host reads those
// while the edge weights at hs are computed and plans the index meanwhile: the
// widest reach from an extent kernel after the edge weights, with its own wait,
// left the GPU idle for about 10 us a likelihood (a search on 50,000 points 22.4
// -> 22.1 ms, on 10,000 5.75 -> 5.22, on 400 3.03 -> 2.63).
constexpr int kMaxHCtas = 512;
__global__ void __launch_bounds__(256) k_adaptive_h(int64_t n, const double* __restrict__ den0,
                                                    const double* __restrict__ logsum, float h, float alpha,
                                                    float* __restrict__ hs, unsigned* hmax) {
    __shared__ unsigned sh[8];
    const double gml = exp(logsum[0] / (double)n);
    unsigned m = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float v = (float)((double)h * pow(den0[i] / gml, (double)alpha));
        hs[i] = v;
        m = max(m, mgk_f2ord(v));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) m = max(m, sh[w]);
        hmax[blockIdx.x] = m;
    }
}

// Per bin: 9 h^2 of its widest point.  r2 starts at -1 (an empty bin), and
// non-negative floats order as their bits, so the maximum is an integer one
// (a thread per bin walking its points took 25 us, the densest bin's chain).
__global__ void k_bin_reach2(int64_t n, const MgkPt* __restrict__ pts, double ox, double oy, double inv_side,
                             int64_t nbx, int64_t nby, float* __restrict__ r2) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const MgkPt p = pts[i];
    int64_t bx = (int64_t)floor(((double)(p.xh + p.xl) - ox) * inv_side);
    int64_t by = (int64_t)floor(((double)(p.yh + p.yl) - oy) * inv_side);
    bx = bx < 0 ? 0 : (bx >= nbx ? nbx - 1 : bx);
    by = by < 0 ? 0 : (by >= nby ? nby - 1 : by);
    atomicMax(reinterpret_cast<int*>(r2) + by * nbx + bx, __float_as_int(9.0f * p.hh));
}

__global__ void k_fill_f32(int64_t n, float v, float* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = v;
}

// Counters of a likelihood computation: context counter slots 5 (edge-mask
// cells) and 6 (point pairs inside the cutoff), accumulated over all steps.
unsigned long long* edge_count(mgk_ctx* c) { return c->d_counter + 5; }
unsigned long long* pair_count(mgk_ctx* c) { return c->d_counter + 6; }

int count_begin(mgk_ctx* c) {
    MGK_CHECK_CUDA(c, cudaMemsetAsync(c->d_counter + 5, 0, 2 * sizeof(unsigned long long), c->stream));
    MGK_CHECK_CUDA(c, cudaEventRecord(c->ev_a, c->stream));
    return MGK_OK;
}

// Reads the counters and the time since count_begin into the context
// (mgk_ctx_last_loo_evals / mgk_ctx_last_loo_ms).
int count_end(mgk_ctx* c) {
    MGK_CHECK_CUDA(c, cudaEventRecord(c->ev_b, c->stream));
    MGK_CHECK_CUDA(c, cudaMemcpyAsync(c->h_counter + 5, c->d_counter + 5, 2 * sizeof(unsigned long long),
                                      cudaMemcpyDeviceToHost, c->stream));
    MGK_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
    c->last_loo_evals[0] = (int64_t)c->h_counter[5];
    c->last_loo_evals[1] = (int64_t)c->h_counter[6];
    MGK_CHECK_CUDA(c, cudaEventElapsedTime(&c->last_loo_ms, c->ev_a, c->ev_b));
    return MGK_OK;
}

// The points in the order in which they are queried, once per search (they do
// not move), and the places of their records in the index at hand; null
// for few points, or without the memory for both: the order of the records.  A
// later step that lacks memory gets theirs (needing).
struct QueryOrder {
    mgk_ctx* c = nullptr;
    int64_t n = 0;
    int32_t *order = nullptr, *inv = nullptr;
    size_t bytes() const { return sizeof(int32_t) * (size_t)std::max<int64_t>(n, 1); }
    void make(mgk_ctx* ctx, const mgk_points* p, const mgk_extent& extent) {
        if (p->n < kPdCurve) return;
        c = ctx;
        n = p->n;
        if (mgk_alloc(c, (void**)&order, bytes()) || mgk_alloc(c, (void**)&inv, bytes()) ||
            mgk_points_curve_order(c, p, extent, order))
            release();
    }
    void release() {
        if (order) mgk_free(c, order, bytes());
        if (inv) mgk_free(c, inv, bytes());
        order = inv = nullptr;
    }
    ~QueryOrder() { release(); }
    // step(), again without the order if it lacked memory (it has launched nothing then)
    template <typename Step>
    int needing(const Step& step) {
        const int st = step();
        if (st != MGK_ERR_BUDGET || !order) return st;
        release();
        return step();
    }
};

// den[input order] and logsum[0] = sum_j log(max(den_j, floor_v)).
// A fixed-h index: every query itself included; per-point h: without it.
int point_density(mgk_ctx* c, const mgk_index* idx, QueryOrder& qo, double* d_den, double floor_v, double* d_logsum) {
    cudaStream_t s = c->stream;
    const int64_t g = (idx->n + kPdQ - 1) / kPdQ;
    if (g == 0) {
        MGK_CHECK_CUDA(c, cudaMemsetAsync(d_logsum, 0, sizeof(double), s));
        return MGK_OK;
    }
    // bin rows split over enough warps to keep every SM busy to the end
    int nsplit = (int)std::min<int64_t>(24, std::max<int64_t>(1, (kPdWarps * (int64_t)c->sm_count + g - 1) / g));
    const int64_t gc = (idx->n + kPdC - 1) / kPdC;
    const int64_t nbins = idx->varh ? idx->nbx * idx->nby : 0;
    const size_t b_part = sizeof(double) * (size_t)gc, b_r2 = sizeof(float) * (size_t)std::max<int64_t>(nbins, 1);
    size_t b_psum = 0;
    double *part = nullptr, *psum = nullptr;
    float* r2 = nullptr;
    auto scratch = [&] {
        part = psum = nullptr;
        b_psum = sizeof(double) * (size_t)idx->n * (size_t)nsplit;
        int st = mgk_alloc(c, (void**)&part, b_part);
        if (st == MGK_OK) st = mgk_alloc(c, (void**)&psum, b_psum);
        if (st == MGK_OK && idx->varh) st = mgk_alloc(c, (void**)&r2, b_r2);
        if (st) {
            mgk_free(c, part, b_part);
            mgk_free(c, psum, b_psum);
        }
        return st;
    };
    int st = qo.needing(scratch);
    while (st == MGK_ERR_BUDGET && nsplit > 1) {  // fewer warps a group then
        nsplit /= 2;
        st = scratch();
    }
    if (st) return st;
    const dim3 grid((unsigned)g, (unsigned)nsplit);
    if (idx->varh) {
        k_fill_f32<<<(unsigned)((nbins + 255) / 256), 256, 0, s>>>(nbins, -1.0f, r2);
        k_bin_reach2<<<(unsigned)((idx->n + 255) / 256), 256, 0, s>>>(idx->n, idx->pts, idx->ox, idx->oy,
                                                                     1.0 / idx->side, idx->nbx, idx->nby, r2);
        k_point_density<true><<<grid, kPdQ, 0, s>>>(idx->n, idx->pts, idx->bin_start, idx->ox, idx->oy, idx->side,
                                                    idx->nbx, idx->nby, idx->reach, idx->h2, r2, qo.order, qo.inv,
                                                    psum, pair_count(c));
    } else {
        k_point_density<false><<<grid, kPdQ, 0, s>>>(idx->n, idx->pts, idx->bin_start, idx->ox, idx->oy, idx->side,
                                                     idx->nbx, idx->nby, idx->reach, idx->h2, nullptr, qo.order,
                                                     qo.inv, psum, pair_count(c));
    }
    k_pd_combine<<<(unsigned)gc, kPdC, 0, s>>>(idx->n, nsplit, psum, qo.order ? qo.order : idx->perm, idx->varh,
                                              idx->h2, floor_v, d_den, part);
    k_sum_parts<<<1, 256, 0, s>>>(gc, part, d_logsum);
    const cudaError_t e = cudaGetLastError();
    // pooled blocks: a later allocation of them is ordered on the same stream
    mgk_free(c, part, b_part);
    mgk_free(c, psum, b_psum);
    if (r2) mgk_free(c, r2, b_r2);
    if (e != cudaSuccess) return mgk_cuda_fail(c, e, "k_point_density");
    MGK_COUNT_LAUNCH(c, idx->varh ? 5 : 3);
    return MGK_OK;
}

// Pilot densities by bandwidth.  The search evaluates the likelihood at
// (h, alpha) pairs that share h (the centre and its two alpha neighbours),
// and the pilot density with its log sum (steps 1-3 up to the geometric
// mean) depends on h alone, so it is kept for the last few h.
struct PilotCache {
    static constexpr int kEntries = 6;
    mgk_ctx* c = nullptr;
    int64_t n = 0;
    uint32_t hbits[kEntries] = {};
    double* buf[kEntries] = {};  // den0[max(n, 1)], then the log sum
    uint64_t last[kEntries] = {};
    uint64_t tick = 0;
    mgk_extent extent;  // of the points (any h)
    cudaEvent_t have_h = nullptr;  // the bandwidths of a likelihood are computed
    QueryOrder qo;
    size_t bytes() const { return sizeof(double) * (size_t)(std::max<int64_t>(n, 1) + 1); }
    ~PilotCache() {
        for (int i = 0; i < kEntries; i++)
            if (buf[i]) mgk_free(c, buf[i], bytes());
        if (have_h) cudaEventDestroy(have_h);
    }
};

// Steps 1-3 up to the geometric mean for bandwidth h: den0 (input order) and
// its log sum, computed or taken from the cache.
int pilot_density(mgk_ctx* c, mgk_points* p, const mgk_raster* r, float h, PilotCache& pc, double** den0) {
    uint32_t hb;
    memcpy(&hb, &h, sizeof(hb));
    int slot = -1;
    for (int i = 0; i < PilotCache::kEntries; i++)
        if (pc.buf[i] && pc.hbits[i] == hb) slot = i;
    if (slot >= 0) {
        pc.last[slot] = ++pc.tick;
        *den0 = pc.buf[slot];
        return MGK_OK;
    }
    for (int i = 0; i < PilotCache::kEntries; i++)  // a free entry, else the least recently used
        if (slot < 0 || !pc.buf[i] || (pc.buf[slot] && pc.last[i] < pc.last[slot])) slot = i;
    int st;
    if (!pc.buf[slot] && (st = pc.qo.needing([&] { return mgk_alloc(c, (void**)&pc.buf[slot], pc.bytes()); }))) return st;
    pc.hbits[slot] = hb;
    pc.last[slot] = ++pc.tick;
    double* den = pc.buf[slot];
    if (r)
        st = pc.qo.needing([&] {
            return mgk_launch_edge_weights(c, p->n, p->x, p->y, nullptr, h, p->dist2, r, p->ew, edge_count(c));
        });
    else st = mgk_edge_weights_unit(c, p);
    if (st == MGK_OK) {
        p->has_ew = true;
        mgk_index* idx = nullptr;
        st = pc.qo.needing([&] {  // h > 0: fixed-h index
            return mgk_index_build_async(c, p, h, 0.0f, &pc.extent, &idx, pc.qo.inv);
        });
        if (st == MGK_OK) {
            st = point_density(c, idx, pc.qo, den, 0.0, den + std::max<int64_t>(p->n, 1));
            mgk_index_destroy(idx);
        }
    }
    if (st) {
        pc.hbits[slot] = 0;  // not a valid entry
        mgk_free(c, pc.buf[slot], pc.bytes());
        pc.buf[slot] = nullptr;
        return st;
    }
    *den0 = den;
    return MGK_OK;
}

unsigned hmax_ctas(int64_t n) { return (unsigned)std::min<int64_t>(kMaxHCtas, (n + 255) / 256); }

// Steps 1-3: the pilot density at h and hs = h (den0 / gml)^alpha into p->h.
int pilot_bandwidths(mgk_ctx* c, mgk_points* p, const mgk_raster* r, float h, float alpha, PilotCache& pc) {
    double* den0 = nullptr;
    int st = pilot_density(c, p, r, h, pc, &den0);
    if (st == MGK_OK && p->n > 0) {
        k_adaptive_h<<<hmax_ctas(p->n), 256, 0, c->stream>>>(p->n, den0, den0 + p->n, h, alpha, p->h, c->d_map + 64);
        MGK_COUNT_LAUNCH(c, 1);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) st = mgk_cuda_fail(c, e, "adaptive bandwidths");
    }
    return st;
}

// LogLikelihood(h, alpha): steps 1-6.
int loglik_adaptive(mgk_ctx* c, mgk_points* p, const mgk_raster* r, float h, float alpha, double* d_den, double* logl,
                    PilotCache& pc) {
    int st = pilot_bandwidths(c, p, r, h, alpha, pc);
    if (st) return st;
    if (!pc.have_h) MGK_CHECK_CUDA(c, cudaEventCreateWithFlags(&pc.have_h, cudaEventDisableTiming));
    MGK_CHECK_CUDA(c, cudaEventRecord(pc.have_h, c->stream));
    if (r && (st = pc.qo.needing([&] {
            return mgk_launch_edge_weights(c, p->n, p->x, p->y, p->h, 0.0f, p->dist2, r, p->ew, edge_count(c));
        })))
        return st;
    // per-point h; bins of 0.75 h (the geometric mean of hs is h), not of the
    // widest h, so that the per-bin reach can cut the window down
    MGK_CHECK_CUDA(c, cudaEventSynchronize(pc.have_h));
    mgk_extent extent = pc.extent;
    if (p->n > 0) {
        const volatile unsigned* w = c->h_map + 64;
        unsigned m = 0;
        for (unsigned b = 0; b < hmax_ctas(p->n); b++) {
            const unsigned u = w[b];
            m = std::max(m, u);
        }
        extent.hmax = mgk_ord2f(m);
    }
    mgk_index* idx = nullptr;
    if ((st = pc.qo.needing([&] { return mgk_index_build_async(c, p, 0.0f, 0.75f * h, &extent, &idx, pc.qo.inv); })))
        return st;
    double *sum = reinterpret_cast<double*>(c->h_map + 32), *d_sum = reinterpret_cast<double*>(c->d_map + 32);
    st = point_density(c, idx, pc.qo, d_den, (double)MGK_EPS_DENSITY_F, d_sum);
    mgk_index_destroy(idx);
    if (st) return st;
    MGK_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
    *logl = *static_cast<volatile double*>(sum);
    return MGK_OK;
}

// The search writes the bandwidths into p->h.  Points that wrap caller
// memory get a buffer of their own, so the caller's array is never written.
int ensure_h(mgk_ctx* c, mgk_points* p) {
    if (p->h && (p->owns_xywh || p->owns_h)) return MGK_OK;
    float* h = nullptr;
    const int st = mgk_alloc(c, (void**)&h, sizeof(float) * (size_t)std::max<int64_t>(p->n, 1));
    if (st) return st;
    p->h = h;
    if (!p->owns_xywh) p->owns_h = true;
    return MGK_OK;
}

}  // namespace

extern "C" {

int mgk_loglik_adaptive(mgk_ctx* c, mgk_points* p, const mgk_raster* r, float h, float alpha, double* logl) {
    if (!c || !p || !logl || !(h > 0.0f)) return mgk_fail(c, MGK_ERR_INVALID, "loglik_adaptive: bad arguments");
    if (r && !p->has_dist2) return mgk_fail(c, MGK_ERR_INVALID, "loglik_adaptive: run mgk_boundary_dist first");
    if (r && std::isfinite(p->dist2_cap))  // the adaptive bandwidths are not known in advance
        return mgk_fail(c, MGK_ERR_INVALID, "loglik_adaptive: needs the exact boundary distances of mgk_boundary_dist");
    int st;
    if ((st = ensure_h(c, p))) return st;
    double* d_den = nullptr;
    const size_t bd = sizeof(double) * (size_t)std::max<int64_t>(p->n, 1);
    if ((st = mgk_alloc(c, (void**)&d_den, bd))) return st;
    {
        PilotCache pc;
        pc.c = c;
        pc.n = p->n;
        st = mgk_points_extent(c, p, false, &pc.extent);
        if (st == MGK_OK) pc.qo.make(c, p, pc.extent);
        if (st == MGK_OK) st = count_begin(c);
        if (st == MGK_OK) st = loglik_adaptive(c, p, r, h, alpha, d_den, logl, pc);
        if (st == MGK_OK) st = count_end(c);
    }
    mgk_free(c, d_den, bd);
    return st;
}

int mgk_adaptive_bandwidths(mgk_ctx* c, mgk_points* p, const mgk_raster* r, float h0, float* h_opt,
                            float* alpha_opt, double* lmax, int* iterations, float* hs_out) {
    if (!c || !p || !(h0 > 0.0f)) return mgk_fail(c, MGK_ERR_INVALID, "adaptive_bandwidths: bad arguments");
    if (r && !p->has_dist2) return mgk_fail(c, MGK_ERR_INVALID, "adaptive_bandwidths: run mgk_boundary_dist first");
    if (r && std::isfinite(p->dist2_cap))  // the adaptive bandwidths are not known in advance
        return mgk_fail(c, MGK_ERR_INVALID, "adaptive_bandwidths: needs the exact boundary distances of mgk_boundary_dist");
    int st;
    if ((st = ensure_h(c, p))) return st;
    double* d_den = nullptr;
    const size_t bd = sizeof(double) * (size_t)std::max<int64_t>(p->n, 1);
    if ((st = mgk_alloc(c, (void**)&d_den, bd))) return st;
    // hooke_jeeves (kde_cuda_kdtr_tiled.cu:3726-3785): float steps, five likelihoods
    float alpha0 = -0.5f;
    float stepH = h0 / 10;
    float stepA = 0.1f;
    // the likelihoods are kept as floats, the type of the reference's Ls array,
    // so that ties and near-ties compare as they do there
    float L[5] = {0, 0, 0, 0, 0};
    PilotCache pc;
    pc.c = c;
    pc.n = p->n;
    auto ll = [&](float h, float a, float* out) {
        double v = 0.0;
        const int s1 = loglik_adaptive(c, p, r, h, a, d_den, &v, pc);
        *out = (float)v;
        return s1;
    };
    // hj_likelihood (:3677-3720): the centre and the neighbours the last move did not keep
    auto around = [&](int last) {
        int s2 = MGK_OK;
        if (s2 == MGK_OK && last == -1) s2 = ll(h0, alpha0, &L[0]);
        if (s2 == MGK_OK && last != 2) s2 = ll(h0 - stepH, alpha0, &L[1]);
        if (s2 == MGK_OK && last != 1) s2 = ll(h0 + stepH, alpha0, &L[2]);
        if (s2 == MGK_OK && last != 4) s2 = ll(h0, alpha0 + stepA, &L[3]);
        if (s2 == MGK_OK && last != 3) s2 = ll(h0, alpha0 - stepA, &L[4]);
        return s2;
    };
    st = mgk_points_extent(c, p, false, &pc.extent);
    if (st == MGK_OK) pc.qo.make(c, p, pc.extent);
    if (st == MGK_OK) st = count_begin(c);
    if (st == MGK_OK) st = around(-1);
    float Lm = L[0];
    const float sH = stepH / 10, sA = stepA / 10;
    int it = 0;
    while (st == MGK_OK && (stepH > sH || stepA > sA) && (h0 - stepH > 0) && it <= 30) {  // MAX_NUM_ITERATIONS
        int dmax = 0;
        for (int i = 0; i < 5; i++)
            if (L[i] > Lm) {
                Lm = L[i];
                dmax = i;
            }
        if (dmax == 0) {
            stepH = stepH / 2;
            stepA = stepA / 2;
        } else {
            // the reference's moves and its bookkeeping of the kept likelihoods
            // (:3750-3778), the move to +stepA included
            if (dmax == 1) {
                h0 = h0 - stepH;
                L[2] = L[0];
                L[0] = L[1];
            }
            if (dmax == 2) {
                h0 = h0 + stepH;
                L[1] = L[0];
                L[0] = L[2];
            }
            if (dmax == 3) {
                alpha0 = alpha0 + stepA;
                L[3] = L[0];
                L[0] = L[4];
            }
            if (dmax == 4) {
                alpha0 = alpha0 - stepA;
                L[3] = L[0];
                L[0] = L[4];
            }
        }
        st = around(dmax);
        it++;
    }
    // final bandwidths at the optimum (main :566-572)
    if (st == MGK_OK) st = pilot_bandwidths(c, p, r, h0, alpha0, pc);
    if (st == MGK_OK && hs_out && p->n > 0) {
        const cudaError_t e = cudaMemcpyAsync(hs_out, p->h, sizeof(float) * (size_t)p->n, cudaMemcpyDeviceToHost,
                                              c->stream);
        if (e != cudaSuccess) st = mgk_cuda_fail(c, e, "adaptive bandwidths download");
    }
    if (st == MGK_OK) st = count_end(c);
    mgk_free(c, d_den, bd);
    if (st) return st;
    p->has_ew = false;  // the weights left behind belong to the fixed h0; recompute at hs
    if (h_opt) *h_opt = h0;
    if (alpha_opt) *alpha_opt = alpha0;
    if (lmax) *lmax = Lm;
    if (iterations) *iterations = it;
    return MGK_OK;
}

}  // extern "C"
