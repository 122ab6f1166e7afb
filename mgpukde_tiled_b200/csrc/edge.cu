// Exact edge-correction weights (Diggle 1985).
//
// CalcEdgeCorrectionWeights (kde_kernel_kdtr.cu:117-189 fixed h, :192-265
// per-point h) and EdgeCorrectionWeightsExact (kde_cuda_kdtr_tiled.cu:2694-2807):
//   e_p = 1                                  if dist2_p >= 9 h^2
//   e_p = 1 / sum_{valid c, d^2 < 9h^2} K_h(d) cellArea   otherwise
// over the reference's NARROW row/column window (a superset of the 3h disc).
//
// The Gaussian factorises over the raster, K ~ exp(-dx^2/2h^2) exp(-dy^2/2h^2),
// and for one row the in-cutoff cells are one contiguous column interval:
// the FP64 test fl(fl(dx^2) + dy^2) < 9h^2 is monotone in |dx| and the cell
// centres are monotone in the column.  So per (point, h), with the column
// factors' prefix sums Q over the window,
//   sum = sum_rows exp(-dy^2/2h^2) * sum_{valid runs of the row} (Q[b] - Q[a])
// where [a, b) is a run of valid cells clipped to the row's in-cutoff
// interval.  The interval ends come from sqrt(9h^2 - dy^2) in FP32; where one
// lies too near a cell centre for that to decide, the oracle's exact FP64 test
// does (the estimate verified, with a binary search when it misses), so the
// summed cell set and the eval count are exactly the reference's.  Work per
// (point, h) is O(window width + window height) rather than O(width x height);
// the sums are FP64, the factors FP64 (per-point h) or FP32 to about 1e-7
// (fixed h, edge_factor).
//
// One warp per point: the lanes build the prefix table of a chunk of up to
// 1024 window columns in shared memory (a contiguous segment per lane and a
// warp scan of the segment totals), then take the window rows in turn.  A
// list of bandwidths is handled in one launch (the LOO bandwidth search needs
// e_p(h) for every candidate h); the weights for h_k go to row k of the
// output.
#include <algorithm>
#include <cmath>

#include "mgk_internal.cuh"

namespace {

constexpr int kEdgeWarps = 4;     // warps per CTA
constexpr int kEdgeChunk = 1024;  // window columns per prefix table

struct EdgeParams {
    int64_t n;
    const float* x;
    const float* y;
    const float* hpp;    // per-point bandwidths (nh = 1) or null
    const float* hgrid;  // device bandwidth list (nh entries) or null: use hfix
    float hfix;
    int nh;
    const double* dist2;  // may be null: no short-circuit
    mgk_grid g;
    const double *cx, *cy;  // cell centres by column and row
    float margin;           // cells by which a centre may lie off its regular place, and the estimates' rounding
    const int64_t* run_start;
    const int2* runs;
    const int4* row_run;  // per row: its first run (x, y), the number of its runs (z)
    float* ew;  // [nh][ew_stride]
    int64_t ew_stride;
    unsigned long long* evals;
    const int* list;        // with nh = 1: the points within 3h of the boundary, else null (all points)
    const int* list_count;  // its length (device)
    unsigned* queue;        // tasks of the list taken beyond each warp's first batch (zeroed)
};

// One bandwidth with boundary distances: the weight of a point 3h or more
// from the boundary is 1 (a coalesced pass); the others are listed (warp-
// aggregated appends, in no fixed order: each weight depends on its point
// alone) for the integral kernel.
template <bool VARH>
__global__ void k_edge_near(EdgeParams E, int* __restrict__ list, int* __restrict__ count) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    bool near = false;
    if (p < E.n) {
        const float hp = VARH ? E.hpp[p] : (E.hgrid ? E.hgrid[0] : E.hfix);
        if (E.dist2[p] >= MGK_CUT * mgk_h2(hp)) E.ew[p] = 1.0f;
        else near = true;
    }
    const unsigned b = __ballot_sync(0xffffffffu, near);
    if (!b) return;  // warp-uniform
    int base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(b));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (near) list[base + __popc(b & ((1u << lane) - 1u))] = (int)p;
}

__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ int64_t trunc_index(double v) {
    v = fmin(fmax(v, -1.0e15), 1.0e15);
    return (int64_t)trunc(v);
}

// exp(-d2 / 2h^2) for d2 within the cutoff (exponent <= 4.5).  Fixed h:
// 2^-(d2 k2) with the exponent in FP64, split into a float pair, 2^-hi by
// the unbiased FP32 polynomial and a first-order correction for the low part
// (relative error about 1e-7; the weights then meet the 1e-6 density and
// likelihood tolerances).  Per-point h (the adaptive search, whose
// Hooke-Jeeves steps compare nearby likelihoods): the FP64 exp.
// (m2: -1 / (2 h^2).)
template <bool VARH>
__device__ __forceinline__ double edge_factor(double d2, double m2, double k2) {
    if (VARH) return exp(d2 * m2);
    const double a = d2 * k2;
    const float ah = (float)a;
    const float al = (float)(a - (double)ah);
    const float e = mgk_exp2_neg_poly(ah);
    return (double)__fmaf_rn(__fmul_rn(-al, MGK_LN2F), e, e);
}

// The oracle's FP64 cutoff decision for column c of a row at dy^2.
__device__ __forceinline__ bool in_cut(const double* cx, int c, double px, double dy2, double cut) {
    const double dx = __dsub_rn(cx[c], px);
    return __dadd_rn(__dmul_rn(dx, dx), dy2) < cut;
}

// The columns [lo, hi] of [c0, c1] inside the cutoff by the exact test, from
// estimates of the ends (out of line: few rows need it).  Empty: lo > hi.
__device__ __noinline__ int2 exact_interval(const double* cx, int c0, int c1, int lo, int hi, double px, double dy2,
                                            double cut) {
    // the column nearest the point: every non-empty interval holds it
    int a = c0, b = c1 + 1;
    while (a < b) {
        const int m = a + ((b - a) >> 1);
        if (cx[m] >= px) b = m;
        else a = m + 1;
    }
    int cm = a > c1 ? c1 : a;
    if (a > c0 && a <= c1 && __dsub_rn(px, cx[a - 1]) < __dsub_rn(cx[a], px)) cm = a - 1;
    if (!in_cut(cx, cm, px, dy2, cut)) return make_int2(1, 0);
    // in_cut is false..true over [c0, cm] and true..false over [cm, c1]
    a = c0;
    b = cm;
    lo = min(max(lo, c0), cm);
    if (in_cut(cx, lo, px, dy2, cut)) {
        b = lo;
        if (lo == c0 || !in_cut(cx, lo - 1, px, dy2, cut)) a = lo;
    } else {
        a = lo + 1;
    }
    while (a < b) {
        const int m = a + ((b - a) >> 1);
        if (in_cut(cx, m, px, dy2, cut)) b = m;
        else a = m + 1;
    }
    lo = a;
    a = cm;
    b = c1;
    hi = min(max(hi, cm), c1);
    if (in_cut(cx, hi, px, dy2, cut)) {
        a = hi;
        if (hi == c1 || !in_cut(cx, hi + 1, px, dy2, cut)) b = hi;
    } else {
        b = hi - 1;
    }
    while (a < b) {
        const int m = a + ((b - a + 1) >> 1);
        if (in_cut(cx, m, px, dy2, cut)) a = m;
        else b = m - 1;
    }
    return make_int2(lo, a);
}

// What bounds it: the latency of its chains (table loads, FP64 operations,
// conversions at 16 lanes a clock) with 24 warps an SM to hide them.  64
// bandwidths on 200,000 points: 23.6 ms with every interval end tested exactly
// (five FP64 tests a row, each from a cell centre formed anew with three
// conversions), 64-bit columns and one task's four divisions after the other;
// 12.2 ms with the centres and each row's first run from tables, the exact
// test only where FP32 cannot decide (a few rows in a hundred), and the tasks'
// divisions side by side.  One bandwidth of 50 on the 10^6 points: 185 -> 121
// us.
template <bool VARH>
__global__ void __launch_bounds__(kEdgeWarps * 32, 6) k_edge_rows(EdgeParams E) {
    __shared__ double qsum[kEdgeWarps][kEdgeChunk + 1];
    const int lane = threadIdx.x & 31;
    double* Q = qsum[threadIdx.x >> 5];
    const int64_t warp0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const mgk_grid& g = E.g;
    const double xll = g.xll, yll = g.yll, cs = g.cs;
    const float inv_cs = 1.0f / g.cs;
    const double cell_area = (double)(g.cs * g.cs);  // float product, kde_cuda_kdtr_tiled.cu:2698
    const int64_t nlist = E.list ? (int64_t)*E.list_count : E.n;
    const int64_t ntask = nlist * (VARH ? 1 : E.nh);
    unsigned long long cnt_total = 0;
    // Tasks (h by h, the points of one h in a row) in batches of up to 32, as
    // large as leave every warp two or more: each lane prepares one, the
    // divisions and square roots of a batch side by side, then the warp takes
    // those that need the integral in turn.  A list of four tasks a warp and
    // more is handed out by a counter, four batches a warp or more: tasks of
    // per-point or wide h differ (an adaptive search on 50,000 points 22.1 -> 21.7
    // ms; 200,000 points at h = 500 1,390 -> 1,272 us, with eight batches 1,255,
    // but at h = 50 66 instead of 59).  With fewer tasks the counter costs more
    // than it evens out (a search on 10,000 points 5.20 -> 5.31 ms).
    unsigned* queue = E.queue && ntask >= 4 * nwarps ? E.queue : nullptr;
    int batch = 32;
    while (batch > 1 && ntask < (queue ? 4 : 2) * nwarps * batch) batch >>= 1;
    for (int64_t t0 = warp0 * batch; t0 < ntask;) {
        unsigned taken = 0;
        if (queue && lane == 0) taken = atomicAdd(queue, (unsigned)batch);
        bool need = false;
        float* out = nullptr;
        float fpx = 0.0f, fpy = 0.0f, fcol_l = 0.0f;
        int icol_l = 0, cl_l = 0, cu_l = -1;
        int64_t rl_l = 0, ru_l = -1;
        double h2_l = 1.0, k2_l = 0.0, acc_l = 0.0;
        if (lane < batch && t0 + lane < ntask) {
            const int64_t k = (t0 + lane) / nlist, i = (t0 + lane) - k * nlist;
            const int64_t p = E.list ? (int64_t)E.list[i] : i;
            const float hp = VARH ? E.hpp[p] : (E.hgrid ? E.hgrid[k] : E.hfix);
            h2_l = mgk_h2(hp);
            out = E.ew + k * E.ew_stride + p;
            need = !E.dist2 || !(E.dist2[p] >= MGK_CUT * h2_l);  // (a NaN bandwidth gives a NaN weight)
            if (!need) *out = 1.0f;
            if (need) {
                fpx = E.x[p];
                fpy = E.y[p];
                const double px = fpx, py = fpy;
                // the point's place in columns: an integer and a fraction
                const double pcol = fmin(fmax((px - xll) / cs - 0.5, -1.0e9), 1.0e9);
                icol_l = (int)floor(pcol);
                fcol_l = (float)(pcol - (double)icol_l);
                k2_l = MGK_LOG2E / (2.0 * h2_l);
                // NARROW window (kde_cuda_kdtr_tiled.cu_l:2719-2727), truncating casts as in Utilities.h:16-17
                const double reach = 3.0 * (double)hp;
                rl_l = g.nrows - 1 - trunc_index((py + reach - yll) / cs);
                ru_l = g.nrows - 1 - trunc_index((py - reach - yll) / cs);
                rl_l = rl_l < 0 ? 0 : rl_l;
                ru_l = ru_l > g.nrows - 1 ? g.nrows - 1 : ru_l;
                cl_l = (int)mgk_min64(mgk_max64(trunc_index((px - reach - xll) / cs), 0), g.ncols);
                cu_l = (int)mgk_max64(mgk_min64(trunc_index((px + reach - xll) / cs), g.ncols - 1), -1);
            }
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, need); todo; todo &= todo - 1u) {
            const int src = __ffs(todo) - 1;
            const double px = __shfl_sync(0xffffffffu, fpx, src), py = __shfl_sync(0xffffffffu, fpy, src);
            const double h2 = __shfl_sync(0xffffffffu, h2_l, src), k2 = __shfl_sync(0xffffffffu, k2_l, src);
            const double cut = MGK_CUT * h2;
            const double m2 = VARH ? -1.0 / (2.0 * h2) : 0.0;
            const int cl = __shfl_sync(0xffffffffu, cl_l, src), cu = __shfl_sync(0xffffffffu, cu_l, src);
            const int icol = __shfl_sync(0xffffffffu, icol_l, src);
            const float fcol = __shfl_sync(0xffffffffu, fcol_l, src);
            const int64_t rl = __shfl_sync(0xffffffffu, rl_l, src), ru = __shfl_sync(0xffffffffu, ru_l, src);
            double acc = 0.0;
            unsigned long long cnt = 0;
            // (counted from cl: a column beyond the last chunk may not fit 32 bits)
            const int width = rl <= ru ? cu - cl + 1 : 0;
            for (int done = 0; done < width; done += min(kEdgeChunk, width - done)) {
                const int c0 = cl + done, c1 = c0 + min(kEdgeChunk, width - done) - 1;
                const int len = c1 - c0 + 1;
                // the column factors, then their prefix sums: Q[j] = sum of the first j
#pragma unroll 2
                for (int j = lane; j < len; j += 32) {
                    const double dx = __dsub_rn(E.cx[c0 + j], px);
                    Q[j + 1] = edge_factor<VARH>(__dmul_rn(dx, dx), m2, k2);
                }
                __syncwarp();
                const int per = (len + 31) >> 5;
                const int j0 = min(len, lane * per), j1 = min(len, j0 + per);
                double run = 0.0;
                for (int j = j0; j < j1; j++) {
                    run += Q[j + 1];
                    Q[j + 1] = run;
                }
                double off = run;
                for (int o = 1; o < 32; o <<= 1) {
                    const double v = __shfl_up_sync(0xffffffffu, off, o);
                    if (lane >= o) off += v;
                }
                off -= run;  // exclusive prefix of the segment totals
                for (int j = j0; j < j1; j++) Q[j + 1] += off;
                if (lane == 0) Q[0] = 0.0;
                __syncwarp();
                // (the next row's table entries are on their way during a row)
                int4 row_n = make_int4(0, 0, 0, 0);
                double cy_n = 0.0;
                if (rl + lane <= ru) {
                    row_n = E.row_run[rl + lane];
                    cy_n = E.cy[rl + lane];
                }
                for (int64_t r = rl + lane; r <= ru; r += 32) {
                    const int4 row = row_n;  // its first run and their number
                    const double dy = __dsub_rn(cy_n, py);
                    if (r + 32 <= ru) {
                        row_n = E.row_run[r + 32];
                        cy_n = E.cy[r + 32];
                    }
                    const double dy2 = __dmul_rn(dy, dy);
                    if (dy2 >= cut) continue;
                    // the half-chord in columns; the ends' places relative to icol
                    const float tc = sqrt_approx((float)(cut - dy2)) * inv_cs;
                    const float fl = fcol - tc, fh = fcol + tc;
                    const float il = ceilf(fl), ih = floorf(fh);
                    const float m = __fmaf_rn(1e-6f, tc, E.margin);
                    int lo, hi;
                    // (false too where the chord has left FP32 and the differences are NaN)
                    if (il - fl >= m && il - fl <= 1.0f - m && fh - ih >= m && fh - ih <= 1.0f - m && tc >= 2.0f * m) {
                        lo = max(icol + (int)il, c0);
                        hi = min(icol + (int)ih, c1);
                    } else {
                        const int2 ex = exact_interval(E.cx, c0, c1, icol + (int)fmaxf(il, -1.0e9f),
                                                       icol + (int)fminf(ih, 1.0e9f), px, dy2, cut);
                        lo = ex.x;
                        hi = ex.y;
                    }
                    if (lo > hi) continue;
                    // valid runs of the row clipped to [lo, hi]
                    double S = 0.0;
                    auto add = [&](int ra, int rb) {  // the run [ra, rb)
                        ra = max(ra, lo);
                        rb = min(rb - 1, hi);
                        if (ra > rb) return;
                        S += Q[rb - c0 + 1] - Q[ra - c0];
                        cnt += (unsigned)(rb - ra + 1);
                    };
                    if (row.z > 0) add(row.x, row.y);
                    if (row.z > 1 && row.y <= hi) {
                        int64_t q = E.run_start[r] + 1;
                        const int64_t qe = E.run_start[r + 1];
                        if (qe - q > 8) {  // first run ending after lo
                            int64_t x0 = q, x1 = qe;
                            while (x0 < x1) {
                                const int64_t m = x0 + ((x1 - x0) >> 1);
                                if (E.runs[m].y <= lo) x0 = m + 1;
                                else x1 = m;
                            }
                            q = x0;
                        }
                        for (; q < qe; q++) {
                            const int2 rr = E.runs[q];
                            if (rr.x > hi) break;
                            add(rr.x, rr.y);
                        }
                    }
                    if (S != 0.0) acc += edge_factor<VARH>(dy2, m2, k2) * S;
                }
                __syncwarp();
            }
            for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            cnt_total += cnt;
            if (lane == src) acc_l = acc;
        }
        if (need) {
            const double k0 = 1.0 / (h2_l * (double)MGK_TWO_PI_F);
            *out = (float)(1.0 / (acc_l * k0 * cell_area));
        }
        t0 = queue ? nwarps * batch + (int64_t)__shfl_sync(0xffffffffu, taken, 0) : t0 + nwarps * batch;
    }
    if (E.evals) {
        for (int o = 16; o; o >>= 1) cnt_total += __shfl_xor_sync(0xffffffffu, cnt_total, o);
        if (lane == 0 && cnt_total) atomicAdd(E.evals, cnt_total);
    }
}

}  // namespace

int mgk_launch_edge_weights_multi(mgk_ctx* ctx, int64_t n, const float* x, const float* y, const float* hpp,
                                  float hfix, const float* d_hgrid, int nh, const double* dist2,
                                  const mgk_raster* rc, float* ew_out, int64_t ew_stride,
                                  unsigned long long* d_evals) {
    if (n == 0 || nh <= 0) return MGK_OK;
    mgk_raster* r = const_cast<mgk_raster*>(rc);  // the run table is a cache of the mask
    int st;
    if ((st = mgk_raster_runs(ctx, r))) return st;
    EdgeParams E{};
    E.n = n;
    E.x = x;
    E.y = y;
    E.hpp = hpp;
    E.hgrid = d_hgrid;
    E.hfix = hfix;
    E.nh = hpp ? 1 : nh;
    E.dist2 = dist2;
    E.g = r->g;
    E.cx = r->centre_x;
    E.cy = r->centre_y;
    {
        // float centres lie within half an ulp of their regular places, the
        // estimates within a few more and 1e-4 cells (their own rounding)
        const double ext = std::max(std::fabs((double)r->g.xll),
                                    std::fabs((double)r->g.xll + (double)r->g.ncols * (double)r->g.cs));
        E.margin = (float)std::min(1.0, 1e-4 + 4.0 * ext * 0x1p-24 / (double)r->g.cs);
    }
    E.row_run = r->row_run;
    E.run_start = r->run_start;
    E.runs = r->runs;
    E.ew = ew_out;
    E.ew_stride = ew_stride;
    E.evals = d_evals;
    const int threads = kEdgeWarps * 32;
    // a grid-stride kernel: one resident wave, so that no CTA starts its
    // share only after the others have finished theirs
    int occ = 1;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &occ, hpp ? (const void*)k_edge_rows<true> : (const void*)k_edge_rows<false>, threads, 0);
    if (e != cudaSuccess) return mgk_cuda_fail(ctx, e, "edge weights occupancy");
    occ = std::max(occ, 1);
    const int64_t blocks = std::min<int64_t>((int64_t)ctx->sm_count * occ, (n * (int64_t)E.nh + kEdgeWarps - 1) / kEdgeWarps);
    int *list = nullptr, *count = nullptr;
    const size_t b_list = sizeof(int) * (size_t)n;
    const bool listed = E.nh == 1 && dist2 && n < (int64_t)INT32_MAX;
    if (listed) {
        if ((st = mgk_alloc(ctx, (void**)&list, b_list))) return st;
        if ((st = mgk_alloc(ctx, (void**)&count, 2 * sizeof(int)))) {
            mgk_free(ctx, list, b_list);
            return st;
        }
        e = cudaMemsetAsync(count, 0, 2 * sizeof(int), ctx->stream);
        if (e == cudaSuccess) {
            const unsigned gn = (unsigned)((n + 255) / 256);
            if (hpp) k_edge_near<true><<<gn, 256, 0, ctx->stream>>>(E, list, count);
            else k_edge_near<false><<<gn, 256, 0, ctx->stream>>>(E, list, count);
            e = cudaGetLastError();
        }
        E.list = list;
        E.list_count = count;
        E.queue = (unsigned*)(count + 1);
    }
    if (e == cudaSuccess) {
        if (hpp) k_edge_rows<true><<<(unsigned)blocks, threads, 0, ctx->stream>>>(E);
        else k_edge_rows<false><<<(unsigned)blocks, threads, 0, ctx->stream>>>(E);
        e = cudaGetLastError();
    }
    // back to the context's pool; later users are ordered after these kernels on the same stream
    if (listed) {
        mgk_free(ctx, list, b_list);
        mgk_free(ctx, count, 2 * sizeof(int));
    }
    if (e != cudaSuccess) return mgk_cuda_fail(ctx, e, "k_edge_rows");
    MGK_COUNT_LAUNCH(ctx, listed ? 2 : 1);
    return MGK_OK;
}

int mgk_launch_edge_weights(mgk_ctx* ctx, int64_t n, const float* x, const float* y, const float* hpp, float h,
                            const double* dist2, const mgk_raster* r, float* ew_out,
                            unsigned long long* d_evals) {
    return mgk_launch_edge_weights_multi(ctx, n, x, y, hpp, h, nullptr, 1, dist2, r, ew_out, n, d_evals);
}
