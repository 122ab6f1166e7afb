// Study-area boundary and point-to-boundary distances.
//
// dMarkBoundary (kde_kernel_kdtr.cu:1209-1281) marks a valid cell as boundary
// when it lies on the raster's outer ring or any of its 8 neighbours is NoData;
// MarkBoundary (kde_cuda_kdtr_tiled.cu:3956-4069) then keeps only those cells.
// dCalcDist2Boundary (kde_kernel_kdtr.cu:1285-1353) takes, per point, the
// minimum squared distance to every boundary-cell centre; the CPU twin
// (kde_cuda_kdtr_tiled.cu:4092-4133) keeps it in double, DBL_MAX when there is
// no boundary cell.  The distance gates the edge-correction short-circuit
// (weight 1 when dist2 >= 9 h^2), so it is computed exactly as the FP64 CPU
// path does: the minimum of exactly rounded double d^2 values.
//
// Here one pass over the mask marks the boundary, compacts the boundary-cell
// centres and counts the rows' runs of valid cells.  For few points or few
// boundary cells every pair is tried; else the centres are binned on a coarse
// grid (32 x 32 cells per bin), each bin gets the list of the cells that can be
// nearest to a point of it, and each point scans its bin's list.  The minimum is
// order independent, so the result is the brute-force minimum bit for bit.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "mgk_internal.cuh"

namespace {

constexpr int kBinCells = 32;  // boundary bins are kBinCells x kBinCells mask cells

// One warp per mask row.  MARK: boundary flags, and the centres of the
// boundary cells appended to `cells` (one atomic per 32 columns with any;
// count[0]).  Both forms: the row's first run of valid cells [a, b), the number
// of its runs (row_run, start[r]) and their total (count[1]).  The cells of three
// rows become validity bits by ballots, 128 columns at a time and 32 ahead;
// outside the raster counts as NoData, so the outer ring is boundary as in
// kde_kernel_kdtr.cu:1209-1281.  Bound by the chains of loads and ballots of a
// row.  Marking alone took 29 us on 2,500^2 cells with a thread per cell and nine
// loads, counting the runs 20 us more; together 41 us (eight chunks a trip 43).
template <bool MARK>
__global__ void __launch_bounds__(128) k_mask_rows(mgk_grid g, const float* __restrict__ mask,
                                                   uint8_t* __restrict__ out, float2* __restrict__ cells,
                                                   unsigned long long* __restrict__ count,
                                                   int64_t* __restrict__ start, int4* __restrict__ row_run) {
    constexpr int kC = 4;  // chunks of 32 columns per trip
    const int lane = threadIdx.x & 31;
    const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (r >= g.nrows) return;  // warp-uniform
    const float nd = g.nodata;
    const float* row = mask + r * g.ncols;
    // validity bits of chunks 0..kC (kC: the next trip's first) of rows r - 1, r, r + 1
    unsigned v[3][kC + 1];
    auto load = [&](int64_t c0, int k) {
        const int64_t c = c0 + 32 * k + lane;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            if (!MARK && i != 1) continue;
            const int64_t rr = r + i - 1;
            const bool ok = c < g.ncols && rr >= 0 && rr < g.nrows && row[(i - 1) * g.ncols + c] != nd;
            v[i][k] = __ballot_sync(0xffffffffu, ok);
        }
    };
    unsigned carry[3] = {0u, 0u, 0u};  // the last column's validity before the trip
    int64_t nruns = 0, nends = 0;
    int a0 = 0, b0 = 0;
    load(0, 0);
    for (int64_t c0 = 0; c0 < g.ncols; c0 += 32 * kC) {
#pragma unroll
        for (int k = 1; k <= kC; k++) load(c0, k);
#pragma unroll
        for (int k = 0; k < kC; k++) {
            const int64_t c = c0 + 32 * k;
            if (c >= g.ncols) break;
            unsigned all = 0xffffffffu;
            unsigned left = 0, right = 0;  // validity of the neighbours in the row itself
#pragma unroll
            for (int i = 0; i < 3; i++) {
                if (!MARK && i != 1) continue;
                const unsigned l = (v[i][k] << 1) | carry[i], rt = (v[i][k] >> 1) | (v[i][k + 1] << 31);
                carry[i] = v[i][k] >> 31;
                all &= v[i][k] & l & rt;
                if (i == 1) {
                    left = l;
                    right = rt;
                }
            }
            const unsigned here = v[1][k], sm = here & ~left, em = here & ~right;
            if (sm && nruns == 0) a0 = (int)c + __ffs(sm) - 1;
            if (em && nends == 0) b0 = (int)c + __ffs(em);
            nruns += __popc(sm);
            nends += __popc(em);
            if (MARK) {
                const unsigned bits = here & ~all;
                if (c + lane < g.ncols) out[r * g.ncols + c + lane] = (bits >> lane) & 1u;
                if (bits) {
                    unsigned long long base = 0;
                    if (lane == 0) base = atomicAdd(count, (unsigned long long)__popc(bits));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if ((bits >> lane) & 1u)
                        cells[base + __popc(bits & ((1u << lane) - 1u))] =
                            make_float2(mgk_cell_x(g.xll, g.cs, c + lane), mgk_cell_y(g.yll, g.cs, g.nrows, r));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 3; i++) v[i][0] = v[i][kC];
    }
    if (lane == 0) {
        start[r] = nruns;
        row_run[r] = make_int4(a0, b0, (int)nruns, 0);
        if (nruns) atomicAdd(count + 1, (unsigned long long)nruns);
    }
}

struct BinGrid {
    double x0, y0, side;  // lower-left corner of bin (0, 0), bin side in coordinates
    int nbx, nby;
};

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ void bin_of(const BinGrid& B, double x, double y, int& bx, int& by) {
    const double fx = floor((x - B.x0) / B.side), fy = floor((y - B.y0) / B.side);
    bx = clampi((int)fmax(fmin(fx, 1e9), -1e9), 0, B.nbx - 1);
    by = clampi((int)fmax(fmin(fy, 1e9), -1e9), 0, B.nby - 1);
}

__global__ void k_bin_count(int64_t nb, const float2* __restrict__ cells, BinGrid B, int* __restrict__ cnt) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nb) return;
    int bx, by;
    bin_of(B, cells[i].x, cells[i].y, bx, by);
    atomicAdd(&cnt[by * B.nbx + bx], 1);
}

// exclusive scan of n ints in one CTA (n is the boundary-bin count, small)
__global__ void __launch_bounds__(1024) k_scan_small(int* __restrict__ a, int n) {
    __shared__ int part[1024];
    const int t = threadIdx.x;
    const int chunk = (n + 1023) / 1024;
    const int b = t * chunk, e = min(n, b + chunk);
    int s = 0;
    for (int i = b; i < e; i++) s += a[i];
    part[t] = s;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const int v = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int run = t ? part[t - 1] : 0;
    for (int i = b; i < e; i++) {
        const int v = a[i];
        a[i] = run;
        run += v;
    }
    if (t == 1023) a[n] = part[1023];
}

__global__ void k_bin_fill(int64_t nb, const float2* __restrict__ cells, BinGrid B, const int* __restrict__ start,
                           int* __restrict__ cursor, float2* __restrict__ binned) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nb) return;
    int bx, by;
    bin_of(B, cells[i].x, cells[i].y, bx, by);
    const int k = by * B.nbx + bx;
    binned[start[k] + atomicAdd(&cursor[k], 1)] = cells[i];
}

__device__ __forceinline__ void scan_bin(const float2* __restrict__ cells, const int* __restrict__ start, int k,
                                         double px, double py, double& best) {
    for (int j = start[k]; j < start[k + 1]; j++) {
        const float2 c = cells[j];
        const double dx = __dsub_rn((double)c.x, px);
        const double dy = __dsub_rn((double)c.y, py);
        best = fmin(best, __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    }
}

// Bin index of perimeter position i (0 <= i < 8r; i = 0 for r = 0) of the
// square ring r around (bx0, by0); false when that bin is off the grid.
__device__ __forceinline__ bool ring_bin(int r, int i, int bx0, int by0, const BinGrid& B, int& kk) {
    int bx, by;
    if (r == 0) {
        bx = bx0;
        by = by0;
    } else if (i < 2 * r + 1) {
        bx = bx0 - r + i;
        by = by0 - r;
    } else if (i < 4 * r + 2) {
        bx = bx0 - r + (i - 2 * r - 1);
        by = by0 + r;
    } else if (i < 6 * r + 1) {
        bx = bx0 - r;
        by = by0 - r + 1 + (i - 4 * r - 2);
    } else {
        bx = bx0 + r;
        by = by0 - r + 1 + (i - 6 * r - 1);
    }
    if (bx < 0 || by < 0 || bx >= B.nbx || by >= B.nby) return false;
    kk = by * B.nbx + bx;
    return true;
}

// Every pair: the squared distance of each point to the nearest of the cells
// [part of them by blockIdx.y], as the bits of a non-negative double (ordered as
// integers), so that the parts meet in an integer minimum.
__global__ void __launch_bounds__(256) k_dist2_all(int64_t n, const float* __restrict__ x, const float* __restrict__ y,
                                                   int64_t nb, const float2* __restrict__ cells,
                                                   unsigned long long* __restrict__ out) {
    __shared__ float2 sc[256];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const double px = i < n ? x[i] : 0.0, py = i < n ? y[i] : 0.0;
    const int64_t b0 = nb * blockIdx.y / gridDim.y, b1 = nb * (blockIdx.y + 1) / gridDim.y;
    double best = DBL_MAX;
    for (int64_t b = b0; b < b1; b += 256) {
        __syncthreads();
        if (b + threadIdx.x < b1) sc[threadIdx.x] = cells[b + threadIdx.x];
        __syncthreads();
        const int m = (int)mgk_min64(256, b1 - b);
#pragma unroll 4
        for (int j = 0; j < m; j++) {
            const double dx = __dsub_rn((double)sc[j].x, px);
            const double dy = __dsub_rn((double)sc[j].y, py);
            best = fmin(best, __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
        }
    }
    if (i >= n) return;
    const unsigned long long bits = (unsigned long long)__double_as_longlong(best);
    if (gridDim.y == 1) out[i] = bits;
    else atomicMin(out + i, bits);
}

__global__ void k_fill_max(int64_t n, double* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = DBL_MAX;
}

// ---- per-bin candidate lists ------------------------------------------------
// For a point p inside bin b (rectangle R), the nearest boundary cell c* obeys
// d(p, c*) <= UB_b = min_c maxdist(R, c) (the farthest corner of R from the
// best cell), so c* is among the cells with mindist(R, c) <= UB_b.  Each bin
// gets that candidate list once; its points then scan only the list.

__device__ __forceinline__ void bin_rect(const BinGrid& B, int bx, int by, double& x0, double& y0, double& x1,
                                         double& y1) {
    x0 = B.x0 + bx * B.side;
    y0 = B.y0 + by * B.side;
    x1 = x0 + B.side;
    y1 = y0 + B.side;
}

__device__ __forceinline__ double mind2(double x0, double y0, double x1, double y1, double cx, double cy) {
    const double dx = fmax(0.0, fmax(x0 - cx, cx - x1)), dy = fmax(0.0, fmax(y0 - cy, cy - y1));
    return dx * dx + dy * dy;
}

__device__ __forceinline__ double maxd2(double x0, double y0, double x1, double y1, double cx, double cy) {
    const double dx = fmax(fabs(cx - x0), fabs(cx - x1)), dy = fmax(fabs(cy - y0), fabs(cy - y1));
    return dx * dx + dy * dy;
}

// The cells of the bins on ring r around a bin, one f(cell index, in range) per
// lane and step, all lanes taking part: the lanes look up 32 bins of the ring
// side by side, then share each non-empty one's cells.
template <typename F>
__device__ __forceinline__ void ring_cells(const int* __restrict__ start, const BinGrid& B, int bx0, int by0, int r,
                                           int lane, const F& f) {
    const int per = r == 0 ? 1 : 8 * r;
    for (int i0 = 0; i0 < per; i0 += 32) {
        int kk, s0 = 0, s1 = 0;
        if (i0 + lane < per && ring_bin(r, i0 + lane, bx0, by0, B, kk)) {
            s0 = start[kk];
            s1 = start[kk + 1];
        }
        for (unsigned m = __ballot_sync(0xffffffffu, s1 > s0); m; m &= m - 1u) {
            const int src = __ffs(m) - 1;
            const int e = __shfl_sync(0xffffffffu, s1, src);
            for (int j = __shfl_sync(0xffffffffu, s0, src); j < e; j += 32) f(j + lane, j + lane < e);
        }
    }
}

// One warp per bin: near[k], the smallest ring (Chebyshev distance in bins)
// with a non-empty bin; ub[k], the bound UB_b capped at cap2; cnt[k], the number
// of cells within it of the bin.  cap2: only cells within sqrt(cap2) of the bin
// rectangle are listed (points farther than that from every boundary cell get
// a distance above cap2).
__global__ void __launch_bounds__(128) k_bin_bounds(const float2* __restrict__ cells, const int* __restrict__ start,
                                                    BinGrid B, double cap2, int* __restrict__ near,
                                                    double* __restrict__ ub, int* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (k >= B.nbx * B.nby) return;  // warp-uniform
    const int bx0 = k % B.nbx, by0 = k / B.nbx;
    double x0, y0, x1, y1;
    bin_rect(B, bx0, by0, x0, y0, x1, y1);
    const double widen = 1e-6 * B.side;
    x0 -= widen;
    y0 -= widen;
    x1 += widen;
    y1 += widen;
    const int rmax = max(B.nbx, B.nby);
    int found = rmax + 1;
    for (int r = 0; r <= rmax; r++) {
        const int per = r == 0 ? 1 : 8 * r;
        bool hit = false;
        for (int i = lane; i < per && !hit; i += 32) {
            int kk;
            hit = ring_bin(r, i, bx0, by0, B, kk) && start[kk + 1] > start[kk];
        }
        if (__any_sync(0xffffffffu, hit)) {
            found = r;
            break;
        }
    }
    // rings whose bins lie within `lim` of this one
    auto within = [&](int r, double lim) {
        const double lb = (double)(r > 0 ? r - 1 : 0) * B.side * (1.0 - 1e-9);
        return r <= rmax && lb * lb <= lim;
    };
    double lim = cap2;
    for (int r = found; within(r, lim); r++) {
        ring_cells(start, B, bx0, by0, r, lane, [&](int j, bool in) {
            if (in) lim = fmin(lim, maxd2(x0, y0, x1, y1, cells[j].x, cells[j].y));
        });
        for (int o = 16; o; o >>= 1) lim = fmin(lim, __shfl_xor_sync(0xffffffffu, lim, o));
    }
    const double cut = lim * (1.0 + 1e-9);
    int n = 0;
    for (int r = found; within(r, cut); r++)
        ring_cells(start, B, bx0, by0, r, lane, [&](int j, bool in) {
            n += in && mind2(x0, y0, x1, y1, cells[j].x, cells[j].y) <= cut;
        });
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) {
        near[k] = found;
        ub[k] = lim;
        cnt[k] = n;
    }
}

// The lists themselves (one warp per bin, in the order of the walk).
__global__ void __launch_bounds__(128) k_bin_lists(const float2* __restrict__ cells, const int* __restrict__ start,
                                                   const int* __restrict__ near, BinGrid B,
                                                   const double* __restrict__ ub, const int* __restrict__ cstart,
                                                   float2* __restrict__ cand) {
    const int lane = threadIdx.x & 31;
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (k >= B.nbx * B.nby || cstart[k + 1] == cstart[k]) return;  // warp-uniform
    const int bx0 = k % B.nbx, by0 = k / B.nbx;
    double x0, y0, x1, y1;
    bin_rect(B, bx0, by0, x0, y0, x1, y1);
    const double widen = 1e-6 * B.side;
    x0 -= widen;
    y0 -= widen;
    x1 += widen;
    y1 += widen;
    const int rmax = max(B.nbx, B.nby);
    const double lim = ub[k] * (1.0 + 1e-9);
    int w = cstart[k];
    for (int r = near[k]; r <= rmax; r++) {
        const double lb = (double)(r > 0 ? r - 1 : 0) * B.side * (1.0 - 1e-9);
        if (lb * lb > lim) break;
        ring_cells(start, B, bx0, by0, r, lane, [&](int j, bool in) {
            float2 c = make_float2(0.0f, 0.0f);
            if (in) c = cells[j];
            const bool take = in && mind2(x0, y0, x1, y1, c.x, c.y) <= lim;
            const unsigned m = __ballot_sync(0xffffffffu, take);
            if (take) cand[w + __popc(m & ((1u << lane) - 1u))] = c;
            w += __popc(m);
        });
    }
}

// Points are searched in the order of their bins (a counting sort by bin),
// so the threads of a warp mostly walk one bin's candidate list: the list's
// loads are shared and the loop lengths agree.  Each result is stored by
// point index, so the order changes no value.
// key[i], the point's bin; rank[i], its place among the bin's points (in no
// fixed order).  With a table of all bins in shared memory a CTA counts its
// 2,048 points there and takes each bin's places with one global atomic
// (800,000 clustered points, 1,900 bins: 59 us with an atomic per point, 16 so).
constexpr int kPointBinsMax = 10240;
template <bool TABLE>
__global__ void __launch_bounds__(256) k_point_bins(int64_t n, const float* __restrict__ x, const float* __restrict__ y,
                                                    BinGrid B, int* __restrict__ key, int* __restrict__ rank,
                                                    int* __restrict__ cnt) {
    extern __shared__ int table[];  // TABLE: the CTA's counts by bin, then the bins' first places
    constexpr int kPts = 8;
    const int nb = B.nbx * B.nby;
    if (TABLE) {
        for (int k = threadIdx.x; k < nb; k += 256) table[k] = 0;
        __syncthreads();
    }
    int kk[kPts], rr[kPts];
    const int64_t i0 = blockIdx.x * (int64_t)(256 * kPts) + threadIdx.x;
#pragma unroll
    for (int j = 0; j < kPts; j++) {
        const int64_t i = i0 + 256 * j;
        kk[j] = -1;
        if (i >= n) continue;
        int bx, by;
        bin_of(B, x[i], y[i], bx, by);
        kk[j] = by * B.nbx + bx;
        rr[j] = atomicAdd(TABLE ? &table[kk[j]] : &cnt[kk[j]], 1);
    }
    if (TABLE) {
        __syncthreads();
        for (int k = threadIdx.x; k < nb; k += 256)
            if (table[k]) table[k] = atomicAdd(&cnt[k], table[k]);
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < kPts; j++) {
        if (kk[j] < 0) continue;
        key[i0 + 256 * j] = kk[j];
        rank[i0 + 256 * j] = rr[j] + (TABLE ? table[kk[j]] : 0);
    }
}

__global__ void k_point_order(int64_t n, const int* __restrict__ key, const int* __restrict__ rank,
                              const int* __restrict__ start, int32_t* __restrict__ order) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) order[start[key[i]] + rank[i]] = (int32_t)i;
}

__global__ void k_dist2_cands(int64_t n, const int32_t* __restrict__ order, const float* __restrict__ x,
                              const float* __restrict__ y, const float2* __restrict__ cells,
                              const int* __restrict__ start, const int* __restrict__ near,
                              const float2* __restrict__ cand, const int* __restrict__ cstart, BinGrid B,
                              double* __restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int64_t i = order ? order[t] : t;
    const double px = x[i], py = y[i];
    double best = DBL_MAX;
    const double fx = floor((px - B.x0) / B.side), fy = floor((py - B.y0) / B.side);
    if (fx >= 0.0 && fy >= 0.0 && fx < (double)B.nbx && fy < (double)B.nby) {
        const int k = (int)fy * B.nbx + (int)fx;
        for (int j = cstart[k]; j < cstart[k + 1]; j++) {
            const float2 c = cand[j];
            const double dx = __dsub_rn((double)c.x, px);
            const double dy = __dsub_rn((double)c.y, py);
            best = fmin(best, __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
        }
        out[i] = best;
        return;
    }
    // outside the bin grid: ring search from the nearest bin
    int bx0, by0;
    bin_of(B, px, py, bx0, by0);
    const int rmax = max(B.nbx, B.nby);
    for (int r = near[by0 * B.nbx + bx0]; r <= rmax; r++) {
        const int ylo = by0 - r, yhi = by0 + r, xlo = bx0 - r, xhi = bx0 + r;
        for (int bx = max(xlo, 0); bx <= min(xhi, B.nbx - 1); bx++) {
            if (ylo >= 0) scan_bin(cells, start, ylo * B.nbx + bx, px, py, best);
            if (r > 0 && yhi < B.nby) scan_bin(cells, start, yhi * B.nbx + bx, px, py, best);
        }
        for (int by = max(ylo + 1, 0); by <= min(yhi - 1, B.nby - 1); by++) {
            if (r > 0 && xlo >= 0) scan_bin(cells, start, by * B.nbx + xlo, px, py, best);
            if (r > 0 && xhi < B.nbx) scan_bin(cells, start, by * B.nbx + xhi, px, py, best);
        }
        const double lb = (double)r * B.side * (1.0 - 1e-9);
        if (best <= lb * lb) break;
    }
    out[i] = best;
}

// The runs of the rows with more than one, at the rows' offsets as half-open
// [a, b): a run starts at a valid cell whose left neighbour is NoData (or the
// row's first cell) and ends after a valid cell whose right neighbour is
// NoData (or the row's last cell).  One warp per row; a single run is in row_run.
__global__ void k_row_runs(mgk_grid g, const float* __restrict__ mask, const int4* __restrict__ row_run,
                           const int64_t* __restrict__ start, int2* __restrict__ runs) {
    const int lane = threadIdx.x & 31;
    const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (r >= g.nrows || row_run[r].z <= 1) return;  // warp-uniform
    const float* row = mask + r * g.ncols;
    const float nd = g.nodata;
    int64_t ns = start[r], ne = ns;
    constexpr int kC = 8;  // chunks of 32 columns whose loads are in flight together
    unsigned v[kC + 1], carry = 0u;
    auto load = [&](int64_t c0, int k) {
        const int64_t c = c0 + 32 * k + lane;
        v[k] = __ballot_sync(0xffffffffu, c < g.ncols && row[c] != nd);
    };
    load(0, 0);
    for (int64_t c0 = 0; c0 < g.ncols; c0 += 32 * kC) {
#pragma unroll
        for (int k = 1; k <= kC; k++) load(c0, k);
#pragma unroll
        for (int k = 0; k < kC; k++) {
            const unsigned sm = v[k] & ~((v[k] << 1) | carry), em = v[k] & ~((v[k] >> 1) | (v[k + 1] << 31));
            const unsigned lt = (1u << lane) - 1u;
            const int c = (int)(c0 + 32 * k) + lane;
            if ((sm >> lane) & 1u) runs[ns + __popc(sm & lt)].x = c;
            if ((em >> lane) & 1u) runs[ne + __popc(em & lt)].y = c + 1;
            ns += __popc(sm);
            ne += __popc(em);
            carry = v[k] >> 31;
        }
        v[0] = v[kC];
    }
}

// The cell centres, as doubles of their float values.
__global__ void k_centres(mgk_grid g, double* __restrict__ cx, double* __restrict__ cy) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < g.ncols) cx[i] = (double)mgk_cell_x(g.xll, g.cs, i);
    else if (i < g.ncols + g.nrows) cy[i - g.ncols] = (double)mgk_cell_y(g.yll, g.cs, g.nrows, i - g.ncols);
}

// Exclusive scan of n int64 values in one CTA; the total goes to a[n].
__global__ void __launch_bounds__(1024) k_scan_i64(int64_t* __restrict__ a, int64_t n) {
    __shared__ int64_t part[1024];
    const int t = threadIdx.x;
    const int64_t chunk = (n + 1023) / 1024;
    const int64_t b = t * chunk, e = mgk_min64(n, b + chunk);
    int64_t s = 0;
    for (int64_t i = b; i < e; i++) s += a[i];
    part[t] = s;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const int64_t v = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int64_t run = t ? part[t - 1] : 0;
    for (int64_t i = b; i < e; i++) {
        const int64_t v = a[i];
        a[i] = run;
        run += v;
    }
    if (t == 1023) a[n] = part[1023];
}

}  // namespace

static BinGrid bin_grid(const mgk_raster* r) {
    return BinGrid{(double)r->g.xll, (double)r->g.yll, (double)kBinCells * (double)r->g.cs, r->bnx, r->bny};
}

// The pass over the mask: the rows' runs, with mark also the boundary.
static int mask_pass(mgk_ctx* ctx, mgk_raster* r, bool mark) {
    const mgk_grid g = r->g;
    cudaStream_t s = ctx->stream;
    mgk_free(ctx, r->run_start, sizeof(int64_t) * (size_t)(g.nrows + 1));
    mgk_free(ctx, r->runs, sizeof(int2) * (size_t)std::max<int64_t>(r->nruns, 1));
    r->run_start = nullptr;
    r->runs = nullptr;
    r->nruns = 0;
    r->has_runs = false;
    if (mark) {  // until the new cells are there the raster is unmarked: a failure leaves no count without cells
        mgk_free(ctx, r->bcells, sizeof(float2) * (size_t)std::max<int64_t>(r->nb, 1));
        r->bcells = nullptr;
        r->nb = 0;
        r->marked = r->binned = false;
        r->cand_cap = -1.0;  // the lists are built by the distance search, for its reach
    }
    if (g.ncols > (int64_t)INT32_MAX - 1) return mgk_fail(ctx, MGK_ERR_INVALID, "raster wider than 2^31 - 2 columns");
    const size_t ncell = (size_t)g.ncols * (size_t)g.nrows;
    int st;
    if (mark && !r->boundary && (st = mgk_alloc(ctx, (void**)&r->boundary, ncell))) return st;
    if ((st = mgk_alloc(ctx, (void**)&r->run_start, sizeof(int64_t) * (size_t)(g.nrows + 1)))) return st;
    if (!r->row_run) {
        const size_t nc = (size_t)(g.ncols + g.nrows);
        if ((st = mgk_alloc(ctx, (void**)&r->row_run, mgk_row_tables_bytes(g)))) return st;
        r->centre_x = reinterpret_cast<double*>(r->row_run + g.nrows);
        r->centre_y = r->centre_x + g.ncols;
        k_centres<<<(unsigned)((nc + 255) / 256), 256, 0, s>>>(g, r->centre_x, r->centre_y);  // of the grid alone
        MGK_CHECK_LAUNCH(ctx, "k_centres");
        MGK_COUNT_LAUNCH(ctx, 1);
    }
    float2* cells = nullptr;
    if (mark && (st = mgk_alloc(ctx, (void**)&cells, sizeof(float2) * ncell))) return st;
    const unsigned grid = (unsigned)((g.nrows * 32 + 127) / 128);
    cudaError_t e = cudaMemsetAsync(ctx->d_counter, 0, 2 * sizeof(unsigned long long), s);
    if (e == cudaSuccess) {
        if (mark)
            k_mask_rows<true><<<grid, 128, 0, s>>>(g, r->mask, r->boundary, cells, ctx->d_counter, r->run_start, r->row_run);
        else
            k_mask_rows<false><<<grid, 128, 0, s>>>(g, r->mask, nullptr, nullptr, ctx->d_counter, r->run_start, r->row_run);
        k_scan_i64<<<1, 1024, 0, s>>>(r->run_start, g.nrows);
        e = cudaGetLastError();
        MGK_COUNT_LAUNCH(ctx, 2);
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(ctx->h_counter, ctx->d_counter, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) st = mgk_cuda_fail(ctx, e, "mask rows");
    const int64_t nb = e == cudaSuccess ? (int64_t)ctx->h_counter[0] : 0;
    const int64_t total = e == cudaSuccess ? (int64_t)ctx->h_counter[1] : 0;
    if (mark && st == MGK_OK) {
        // bins of kBinCells x kBinCells mask cells over the mask extent
        if (!r->bstart) {
            r->bnx = (int)((g.ncols + kBinCells - 1) / kBinCells);
            r->bny = (int)((g.nrows + kBinCells - 1) / kBinCells);
            r->nbins = (int64_t)r->bnx * r->bny;
        }
        st = mgk_alloc(ctx, (void**)&r->bcells, sizeof(float2) * (size_t)std::max<int64_t>(nb, 1));
        if (st == MGK_OK) r->nb = nb;
        if (st == MGK_OK && nb > 0 &&
            (e = cudaMemcpyAsync(r->bcells, cells, sizeof(float2) * (size_t)nb, cudaMemcpyDeviceToDevice, s)) != cudaSuccess)
            st = mgk_cuda_fail(ctx, e, "boundary cells");
        if (st == MGK_OK) r->marked = true;
    }
    if (cells) mgk_free(ctx, cells, sizeof(float2) * ncell);  // later users are ordered after the copy
    if (st) return st;
    if ((st = mgk_alloc(ctx, (void**)&r->runs, sizeof(int2) * (size_t)std::max<int64_t>(total, 1)))) return st;
    r->nruns = total;
    if (total > 0) {
        k_row_runs<<<grid, 128, 0, s>>>(g, r->mask, r->row_run, r->run_start, r->runs);
        MGK_CHECK_LAUNCH(ctx, "k_row_runs");
        MGK_COUNT_LAUNCH(ctx, 1);
    }
    r->has_runs = true;
    return MGK_OK;
}

int mgk_raster_runs(mgk_ctx* ctx, mgk_raster* r) { return r->has_runs ? MGK_OK : mask_pass(ctx, r, false); }

int mgk_launch_mark_boundary(mgk_ctx* ctx, mgk_raster* r) { return mask_pass(ctx, r, true); }

// The boundary cells into their bins.
static int bin_cells(mgk_ctx* ctx, mgk_raster* r) {
    cudaStream_t s = ctx->stream;
    const size_t b_cells = sizeof(float2) * (size_t)std::max<int64_t>(r->nb, 1);
    const size_t b_start = sizeof(int) * (size_t)(r->nbins + 1);
    float2* binned = nullptr;
    int* cursor = nullptr;
    int st;
    if ((!r->bstart && (st = mgk_alloc(ctx, (void**)&r->bstart, b_start))) ||
        (!r->bnear && (st = mgk_alloc(ctx, (void**)&r->bnear, b_start))) ||
        (st = mgk_alloc(ctx, (void**)&binned, b_cells)))
        return st;
    if ((st = mgk_alloc(ctx, (void**)&cursor, b_start))) {
        mgk_free(ctx, binned, b_cells);
        return st;
    }
    const BinGrid B = bin_grid(r);
    const unsigned gb = (unsigned)((r->nb + 255) / 256);
    cudaError_t e = cudaMemsetAsync(r->bstart, 0, b_start, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(cursor, 0, b_start, s);
    if (e == cudaSuccess) {
        k_bin_count<<<gb, 256, 0, s>>>(r->nb, r->bcells, B, r->bstart);
        k_scan_small<<<1, 1024, 0, s>>>(r->bstart, (int)r->nbins);
        k_bin_fill<<<gb, 256, 0, s>>>(r->nb, r->bcells, B, r->bstart, cursor, binned);
        e = cudaGetLastError();
        MGK_COUNT_LAUNCH(ctx, 3);
    }
    mgk_free(ctx, cursor, b_start);  // later users are ordered after these kernels
    if (e != cudaSuccess) {
        mgk_free(ctx, binned, b_cells);
        return mgk_cuda_fail(ctx, e, "boundary bins");
    }
    mgk_free(ctx, r->bcells, b_cells);
    r->bcells = binned;
    r->binned = true;
    return MGK_OK;
}

// Per-bin candidate lists for distances exact up to `cap` (coordinate units;
// infinite: every distance exact).  Bins whose nearest boundary cells lie
// beyond the cap get short or empty lists, so a small cap (3h: what the
// edge-weight short-circuit asks) makes the lists and the search cheap.
static int build_cands(mgk_ctx* ctx, mgk_raster* r, double cap) {
    cudaStream_t s = ctx->stream;
    int st;
    if (!r->binned && (st = bin_cells(ctx, r))) return st;
    const BinGrid B = bin_grid(r);
    const size_t b_start = sizeof(int) * (size_t)(r->nbins + 1);
    const double cap2 = std::isfinite(cap) ? cap * cap * (1.0 + 1e-9) : DBL_MAX;
    if (r->bub) mgk_free(ctx, r->bub, sizeof(double) * (size_t)r->nbins);
    if (r->cstart) mgk_free(ctx, r->cstart, b_start);
    if (r->cand) mgk_free(ctx, r->cand, sizeof(float2) * (size_t)std::max<int64_t>(r->ncand, 1));
    r->bub = nullptr;
    r->cstart = nullptr;
    r->cand = nullptr;
    r->ncand = 0;
    r->cand_cap = -1.0;
    if ((st = mgk_alloc(ctx, (void**)&r->bub, sizeof(double) * (size_t)r->nbins)) ||
        (st = mgk_alloc(ctx, (void**)&r->cstart, b_start)))
        return st;
    const unsigned gbin = (unsigned)((r->nbins * 32 + 127) / 128);  // one warp per bin
    k_bin_bounds<<<gbin, 128, 0, s>>>(r->bcells, r->bstart, B, cap2, r->bnear, r->bub, r->cstart);
    k_scan_small<<<1, 1024, 0, s>>>(r->cstart, (int)r->nbins);
    MGK_CHECK_LAUNCH(ctx, "boundary candidate lists");
    MGK_COUNT_LAUNCH(ctx, 2);
    int total = 0;
    MGK_CHECK_CUDA(ctx, cudaMemcpyAsync(&total, r->cstart + r->nbins, sizeof(int), cudaMemcpyDeviceToHost, s));
    MGK_CHECK_CUDA(ctx, cudaStreamSynchronize(s));
    r->ncand = total;
    if ((st = mgk_alloc(ctx, (void**)&r->cand, sizeof(float2) * (size_t)std::max(total, 1)))) return st;
    if (total > 0) {
        k_bin_lists<<<gbin, 128, 0, s>>>(r->bcells, r->bstart, r->bnear, B, r->bub, r->cstart, r->cand);
        MGK_CHECK_LAUNCH(ctx, "boundary candidate fill");
        MGK_COUNT_LAUNCH(ctx, 1);
    }
    r->cand_cap = std::isfinite(cap) ? cap : INFINITY;
    return MGK_OK;
}

int mgk_launch_dist2(mgk_ctx* ctx, mgk_points* p, mgk_raster* r, double cap) {
    cudaStream_t s = ctx->stream;
    const int64_t n = p->n;
    if (n == 0) return MGK_OK;
    const unsigned gp = (unsigned)((n + 255) / 256);
    if (r->nb == 0) {
        k_fill_max<<<gp, 256, 0, s>>>(n, p->dist2);
        MGK_CHECK_LAUNCH(ctx, "k_fill_max");
        MGK_COUNT_LAUNCH(ctx, 1);
        return MGK_OK;
    }
    // Every pair up to 2^26 of them: 10 us for 2,000 points and 500 cells, 36 us
    // for 20,000 and 3,000, in one kernel.  The lists take eight kernels and a
    // wait (115 us of kernels for those 2,000 points, 150 us for the 20,000), but
    // hardly more for ten times the pairs.
    if (!(r->cand_cap >= cap) && (double)n * (double)r->nb <= 0x1p26) {
        const unsigned parts = (unsigned)std::max<int64_t>(
            1, std::min<int64_t>((r->nb + 255) / 256, 4 * (int64_t)ctx->sm_count / (int64_t)gp));
        cudaError_t e = cudaSuccess;
        // the largest integer: above DBL_MAX, which a point at infinity or NaN keeps
        if (parts > 1) e = cudaMemsetAsync(p->dist2, 0xff, sizeof(double) * (size_t)n, s);
        if (e == cudaSuccess) {
            k_dist2_all<<<dim3(gp, parts), 256, 0, s>>>(n, p->x, p->y, r->nb, r->bcells,
                                                       reinterpret_cast<unsigned long long*>(p->dist2));
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) return mgk_cuda_fail(ctx, e, "k_dist2_all");
        MGK_COUNT_LAUNCH(ctx, 1);
        return MGK_OK;
    }
    if (!(r->cand_cap >= cap)) {  // no lists yet, or lists for a shorter reach
        int st = build_cands(ctx, r, cap);
        if (st) return st;
    }
    const BinGrid B = bin_grid(r);
    if (n >= (int64_t)INT32_MAX) {
        k_dist2_cands<<<gp, 256, 0, s>>>(n, nullptr, p->x, p->y, r->bcells, r->bstart, r->bnear, r->cand, r->cstart, B,
                                         p->dist2);
    } else {
        // counting sort of the points by bin, then the search in that order
        // (the ranks lie in the result array until the search writes it)
        const size_t b_key = sizeof(int) * (size_t)n, b_cnt = sizeof(int) * (size_t)(r->nbins + 1);
        int *key = nullptr, *cnt = nullptr;
        int32_t* order = nullptr;
        int st;
        if ((st = mgk_alloc(ctx, (void**)&key, b_key))) return st;
        if ((st = mgk_alloc(ctx, (void**)&order, b_key)) || (st = mgk_alloc(ctx, (void**)&cnt, b_cnt))) {
            mgk_free(ctx, key, b_key);
            mgk_free(ctx, order, b_key);
            return st;
        }
        int* rank = reinterpret_cast<int*>(p->dist2);
        cudaError_t e = cudaMemsetAsync(cnt, 0, b_cnt, s);
        if (e == cudaSuccess) {
            const unsigned g8 = (unsigned)((n + 2047) / 2048);
            if (r->nbins <= kPointBinsMax)
                k_point_bins<true><<<g8, 256, sizeof(int) * (size_t)r->nbins, s>>>(n, p->x, p->y, B, key, rank, cnt);
            else
                k_point_bins<false><<<g8, 256, 0, s>>>(n, p->x, p->y, B, key, rank, cnt);
            k_scan_small<<<1, 1024, 0, s>>>(cnt, (int)r->nbins);
            k_point_order<<<gp, 256, 0, s>>>(n, key, rank, cnt, order);
            k_dist2_cands<<<gp, 256, 0, s>>>(n, order, p->x, p->y, r->bcells, r->bstart, r->bnear, r->cand, r->cstart,
                                             B, p->dist2);
            e = cudaGetLastError();
        }
        // the buffers go back to the context's pool; later users are ordered
        // after these kernels on the same stream
        mgk_free(ctx, key, b_key);
        mgk_free(ctx, order, b_key);
        mgk_free(ctx, cnt, b_cnt);
        if (e != cudaSuccess) return mgk_cuda_fail(ctx, e, "k_dist2");
        MGK_COUNT_LAUNCH(ctx, 3);
    }
    MGK_CHECK_LAUNCH(ctx, "k_dist2");
    MGK_COUNT_LAUNCH(ctx, 1);
    return MGK_OK;
}
