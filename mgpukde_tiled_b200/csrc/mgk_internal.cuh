// Internal declarations shared by the CUDA translation units of libmgk.
#pragma once
#include <cstring>

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <map>
#include <string>
#include <vector>

#include "../../include/mgk.h"

// ---- constants of the reference (Utilities.h) -----------------------------
// TWO_PI is a float constant in the reference (Utilities.h:8).
#define MGK_TWO_PI_F 6.2831853071795862f
// EPSILONDENSITY (Utilities.h:20), a float constant.
#define MGK_EPS_DENSITY_F 0.00000000000001f
// CUT_OFF_FACTOR (Utilities.h:27): the kernel is zero for d^2 >= 9 h^2.
#define MGK_CUT 9.0
#define MGK_LOG2E 1.4426950408889634
#define MGK_LN2F 0.69314718055994531f

// ---- host-side objects -----------------------------------------------------
struct mgk_raster_pipe;  // streams and events of the whole-raster path (api.cu)

struct mgk_ctx {
    int device = 0;
    int sm_count = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    uint64_t budget = 0;
    std::atomic<uint64_t> in_use{0};  // read by other threads (serving statistics)
    std::string last_error;
    // small pinned/device scratch for scalar results
    unsigned long long* d_counter = nullptr;  // 8 counters
    unsigned long long* h_counter = nullptr;  // pinned mirror
    // mapped page-locked staging of plans and counts (mgk_host_stage), in
    // kStageSlots independent slots; h_stage[i] and d_stage[i] address the same
    // bytes.  Slot 3 holds the bit-packed density mask of mgk_kde_raster.
    static constexpr int kStageSlots = 4;
    void* h_stage[kStageSlots] = {};
    void* d_stage[kStageSlots] = {};
    size_t h_stage_bytes[kStageSlots] = {};
    // a small mapped page-locked page: words 32 and 33 an adaptive likelihood (a
    // double), words 64.. the extents of k_extent's CTAs or the largest h of
    // k_adaptive_h's
    unsigned *h_map = nullptr, *d_map = nullptr;
    mgk_raster_pipe* pipe = nullptr;
    std::multimap<size_t, void*> pool;        // cached device blocks by size class
    uint64_t launches = 0;                    // kernels launched by this context
    cudaEvent_t ev_a = nullptr, ev_b = nullptr;
    bool marking = false;             // mgk_mark_boundary has been called since the stream was set
    cudaEvent_t ev_marked = nullptr;  // after its kernels, on a caller's stream
    float last_density_ms = 0.0f;
    int64_t last_loo_evals[2] = {0, 0};  // edge and LOO evals of the last LOO batch run
    float last_loo_ms = 0.0f;
    // tuning (mgk_autotune / mgk_ctx_set_tuning)
    float bin_factor = 0.5f;   // default index bin side / h (fastest of 0.5-1.25 on the 1e6-point raster)
    int split_waves = 4;       // density work items per resident CTA slot (4 of 2-32 fastest on the C1 raster)
    int64_t tile_side = 0;     // streamed tile side (0: whole raster when it fits)
};

#define MGK_COUNT_LAUNCH(ctx, k) ((ctx)->launches += (k))

struct mgk_points {
    mgk_ctx* ctx = nullptr;
    int64_t n = 0;
    float *x = nullptr, *y = nullptr, *w = nullptr, *h = nullptr;
    bool owns_xywh = false;
    bool owns_h = false;  // h allocated by the adaptive search on points that do not own x/y/w/h
    double* dist2 = nullptr;
    bool has_dist2 = false;
    // dist2 is exact for the points whose nearest boundary cell lies within
    // dist2_cap (coordinate units); the others hold a value above dist2_cap^2
    double dist2_cap = 0.0;
    float* ew = nullptr;
    bool has_ew = false;
};

struct mgk_raster {
    mgk_ctx* ctx = nullptr;
    mgk_grid g{};
    float* mask = nullptr;
    bool owns = false;
    uint8_t* boundary = nullptr;  // per cell
    float2* bcells = nullptr;     // boundary-cell centres, binned once the lists are built
    bool binned = false;
    int* bstart = nullptr;        // bin offsets into bcells (nbins + 1)
    int* bnear = nullptr;         // per bin: first ring index holding a non-empty bin
    double* bub = nullptr;        // per bin: upper bound of the nearest-cell d^2 of its points
    int* cstart = nullptr;        // per bin: offsets of its candidate list in cand (nbins + 1)
    float2* cand = nullptr;       // candidate boundary-cell centres, bin by bin
    int64_t ncand = 0;
    double cand_cap = -1.0;       // the lists hold the cells within this reach of each bin (< 0: no lists)
    int bnx = 0, bny = 0;         // boundary bins per row / column
    int64_t nbins = 0;
    int64_t nb = 0;
    bool marked = false;
    // valid-cell runs per row: runs[run_start[r] .. run_start[r+1]) = [a, b)
    int64_t* run_start = nullptr;  // nrows + 1
    int2* runs = nullptr;
    int64_t nruns = 0;
    bool has_runs = false;
    // per row its first run (x, y) and the number of its runs (z); cell centres
    // by column and row (one block, mgk_row_tables_bytes)
    int4* row_run = nullptr;
    double *centre_x = nullptr, *centre_y = nullptr;
};
inline size_t mgk_row_tables_bytes(const mgk_grid& g) {
    return sizeof(int4) * (size_t)g.nrows + sizeof(double) * (size_t)(g.ncols + g.nrows);
}

// One point of the bin-major index (32 B, one bulk copy moves whole records).
// Coordinates are split on a global quantum q = 2^-qexp: x = xh + xl exactly,
// xh a multiple of q, |xl| <= q/2.  Cell centres are split on the same
// quantum, so xh - cxh is exact in FP32 and the distance is recovered
// exactly as a float pair.  wk = w * e (fixed h) or w * e / (h^2 TWO_PI)
// (per-point h); k2h + k2l = log2(e) / (2 h^2) and hh = h*h (float product)
// for per-point h, zero otherwise.
struct __align__(16) MgkPt {
    float xh, yh, xl, yl;
    float wk, k2h, k2l, hh;
};

struct mgk_index {
    mgk_ctx* ctx = nullptr;
    int64_t n = 0;
    bool varh = false;
    int qexp = 0;  // coordinate quantum 2^-qexp
    // fixed-h constants (double): h^2 as the reference forms it, 9 h^2,
    // log2(e)/(2 h^2), 1/(h^2 TWO_PI), 3 h
    float h = 0.0f;
    double h2 = 0, cut_d2 = 0, k2 = 0, k0 = 0, reach = 0;
    // bin grid
    double ox = 0, oy = 0, side = 1;
    int64_t nbx = 1, nby = 1;
    int32_t* bin_start = nullptr;  // nbx*nby + 1
    // bin-major point data
    MgkPt* pts = nullptr;
    int32_t* perm = nullptr; // sorted position -> input index
    uint64_t bytes = 0;
};

// ---- helpers ---------------------------------------------------------------
int mgk_fail(mgk_ctx* ctx, int status, const std::string& msg);
int mgk_cuda_fail(mgk_ctx* ctx, cudaError_t e, const char* what);
int mgk_alloc(mgk_ctx* ctx, void** p, size_t bytes);
// Mapped page-locked host memory of at least `bytes` owned by the context
// (grown on demand, previous contents not kept): *host and *dev address the
// same bytes.  Kernels read and write it directly over the bus, so small
// per-launch tables and flags need no copy-engine transfer and never queue
// behind large copies that other streams have in flight.  One user at a time:
// kernels using it must have finished before the next call.
int mgk_host_stage(mgk_ctx* ctx, size_t bytes, void** host, void** dev);
// The same for staging slot `slot` (0 is the one mgk_host_stage uses); plans
// that are alive at the same time use different slots.
int mgk_host_stage_slot(mgk_ctx* ctx, int slot, size_t bytes, void** host, void** dev);
void mgk_free(mgk_ctx* ctx, void* p, size_t bytes);

#define MGK_CHECK_CUDA(ctx, expr)                                   \
    do {                                                            \
        cudaError_t e_ = (expr);                                    \
        if (e_ != cudaSuccess) return mgk_cuda_fail(ctx, e_, #expr); \
    } while (0)

#define MGK_CHECK_LAUNCH(ctx, name)                                   \
    do {                                                              \
        cudaError_t e_ = cudaGetLastError();                          \
        if (e_ != cudaSuccess) return mgk_cuda_fail(ctx, e_, name);   \
    } while (0)

// ---- device helpers --------------------------------------------------------
__device__ __host__ __forceinline__ int64_t mgk_min64(int64_t a, int64_t b) { return a < b ? a : b; }
__device__ __host__ __forceinline__ int64_t mgk_max64(int64_t a, int64_t b) { return a > b ? a : b; }

__device__ __forceinline__ float mgk_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 2^-a for 0 <= a < 120, without the special-function unit: a = n + f with
// n = rint(a), |f| <= 1/2 (Cody-Waite reduction), e^t for t = -f ln 2 from its
// Taylor series to degree 8 (truncation below 2.1e-10 relative for
// |t| <= ln2/2), Horner in FMA, then scaled by 2^-n through the exponent
// bits.  Its rounding errors have no common sign across inputs, so sums of
// many terms carry no systematic bias (used where millions of terms feed one
// logarithm sum).
__device__ __forceinline__ float mgk_exp2_neg_poly(float a) {
    const float n = rintf(a);
    const float t = __fmul_rn(__fsub_rn(n, a), MGK_LN2F);
    float p = 2.4801587301587302e-05f;  // 1/8!
    p = __fmaf_rn(p, t, 1.9841269841269841e-04f);  // 1/7!
    p = __fmaf_rn(p, t, 1.3888888888888889e-03f);  // 1/6!
    p = __fmaf_rn(p, t, 8.3333333333333333e-03f);  // 1/5!
    p = __fmaf_rn(p, t, 4.1666666666666667e-02f);  // 1/4!
    p = __fmaf_rn(p, t, 1.6666666666666667e-01f);  // 1/3!
    p = __fmaf_rn(p, t, 0.5f);
    p = __fmaf_rn(p, t, 1.0f);
    p = __fmaf_rn(p, t, 1.0f);
    return __fmul_rn(p, __int_as_float((127 - (int)n) << 23));
}

// Two FP32 values in a 64-bit register (sm_100 f32x2; each half is
// rounded as the scalar operation is)
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_dup(float a) {
    f2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ f2 f2_make(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_get(f2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// 2^-g for g in [-1/2, 1/2]: a degree-6 polynomial, fitted to 2^-g by least
// squares on Chebyshev nodes with the mean error held where the rounding of
// the terms leaves none, each coefficient rounded to float before the next
// ones are fitted (truncation 3.3e-9 relative).  Terms 2^-a formed with it over
// the cutoff's disc: relative error 7.04e-8 rms, 2.3e-7 at most, at most 2e-11
// in the weighted mean (with the degree-8 Taylor form of mgk_exp2_neg_poly
// 7.05e-8, 2.3e-7, 7e-11).  Scalar with immediate coefficients: a packed FMA
// with three register pairs runs at 3.3 cycles instead of 2.
__device__ __forceinline__ float mgk_exp2_neg_frac(float g) {
    float p = __fmaf_rn(0.00015285507834050804f, g, -0.001339130220003426f);
    p = __fmaf_rn(p, g, 0.009618666023015976f);
    p = __fmaf_rn(p, g, -0.055503588169813156f);
    p = __fmaf_rn(p, g, 0.24022646248340607f);
    p = __fmaf_rn(p, g, -0.6931471824645996f);
    return __fmaf_rn(p, g, 1.0f);
}

__device__ __forceinline__ float mgk_min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Cell centres as the reference computes them (Utilities.h:13-14): double
// arithmetic, stored to float.
__device__ __host__ __forceinline__ float mgk_cell_x(double xll, double cs, int64_t col) {
    return (float)(xll + ((double)col + 0.5) * cs);
}
__device__ __host__ __forceinline__ float mgk_cell_y(double yll, double cs, int64_t nrows, int64_t row) {
    return (float)(yll + ((double)nrows - 0.5 - (double)row) * cs);
}

// Exact squared distance of two float positions with the rounding of the
// FP64 oracle (products and sum each rounded once, never fused).
__device__ __forceinline__ double mgk_d2_exact(float x0, float y0, float x1, float y1) {
    const double dx = __dsub_rn((double)x1, (double)x0);
    const double dy = __dsub_rn((double)y1, (double)y0);
    return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
}

// Splits a float coordinate on the quantum 2^-qexp: hi = nearest multiple,
// lo = remainder, both exact floats (|v| < 2^(22 - qexp) assumed).
// 2^k for a double exponent in the normal range (|k| < 1000), from its bits.
__device__ __host__ __forceinline__ double mgk_pow2(int k) {
    const unsigned long long b = (unsigned long long)(1023 + k) << 52;
    double d;
    memcpy(&d, &b, sizeof d);
    return d;
}
__device__ __host__ __forceinline__ void mgk_qsplit(float v, int qexp, float& hi, float& lo) {
    // scaling by powers of two is exact, so multiplying by 2^-qexp is the
    // division by 2^qexp
    hi = (float)(rint((double)v * mgk_pow2(qexp)) * mgk_pow2(-qexp));
    lo = (float)((double)v - (double)hi);
}

// h^2 exactly as the reference's CPU path forms it: float product widened.
__device__ __host__ __forceinline__ double mgk_h2(float h) {
    const float hh = h * h;
    return (double)hh;
}

// Floats as unsigned integers in the same order, and back.
__device__ __forceinline__ unsigned mgk_f2ord(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
inline float mgk_ord2f(unsigned u) {
    u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    float f;
    memcpy(&f, &u, 4);
    return f;
}

// ---- kernels launched across translation units ------------------------------
struct mgk_extent {
    double xmin = 0, ymin = 0, xmax = 1, ymax = 1;
    float hmax = 0;
};
int mgk_points_extent(mgk_ctx* ctx, const mgk_points* pts, bool want_h, mgk_extent* out);
// Builds the index on ctx->stream without waiting for it; the points' arrays
// are read until it is done.  inv (device, n entries, or
// null): the place of each point's record.
int mgk_launch_index_build(mgk_ctx* ctx, const mgk_points* pts, float h, float bin_size, const mgk_extent* extent,
                           mgk_index* idx, int32_t* inv = nullptr);
// The same into a new index, for callers that wait later on the same stream.
int mgk_index_build_async(mgk_ctx* ctx, const mgk_points* pts, float h, float bin_size, const mgk_extent* extent,
                          mgk_index** out, int32_t* inv = nullptr);
// The points (n entries, device) along a Hilbert curve over their extent, stream-ordered.
int mgk_points_curve_order(mgk_ctx* ctx, const mgk_points* pts, const mgk_extent& extent, int32_t* d_order);
// The index records' weights from the points' current edge weights (an index
// built before the edge weights were known), stream-ordered on ctx->stream.
int mgk_index_refresh_weights(mgk_ctx* ctx, mgk_index* idx, const mgk_points* pts);
// Indexes with bin sides side0 2^l (l < nlev, fewer when the bin-count limit raises a side) and for each
// the positions of its records in Z-order of the bins; what is made before a failure is the caller's to free.
int mgk_index_build_levels(mgk_ctx* ctx, const mgk_points* pts, float h, double side0, int nlev,
                           const mgk_extent* extent, std::vector<mgk_index*>* lev, std::vector<int32_t*>* order);
int mgk_launch_density(mgk_ctx* ctx, const mgk_index* idx, const mgk_grid* g, int64_t row0,
                       int64_t col0, int64_t nr, int64_t nc, const float* d_mask, float* d_out,
                       unsigned long long* d_evals, bool fp64);
int mgk_launch_density_jobs(mgk_ctx* ctx, int njobs, const mgk_tile_job* jobs, unsigned long long* d_evals);
// mgk_launch_density in two halves, so a caller can put its own copies
// between the plan (which synchronises the context stream and uploads the
// work list) and the kernels: prepare plans and uploads; execute launches,
// waits and releases the plan (also on failure); discard releases an unrun
// plan.  One plan at a time per context (the work list shares the context's
// page-locked staging).  A tile with no cells gives a null plan, which
// execute accepts.
struct mgk_dplan;
int mgk_density_prepare(mgk_ctx* ctx, const mgk_index* idx, const mgk_grid* g, int64_t row0, int64_t col0,
                        int64_t nr, int64_t nc, const float* d_mask, float* d_out, unsigned long long* d_evals,
                        bool fp64, mgk_dplan** out);
int mgk_density_execute(mgk_ctx* ctx, mgk_dplan* plan);
void mgk_density_discard(mgk_ctx* ctx, mgk_dplan* plan);
// A tile pipeline that plans tile k + 1 while tile k computes, all on one
// stream: counts_launch queues the counting kernel of a tile into staging
// slot `slot` (it leaves the shared staging-wait flag alone: the caller
// zeroes it once and reads it at the end); once that kernel has finished,
// plan_counted builds the plan from the counts into the same slot; launch
// queues the plan's kernels on stream s without waiting; discard releases the
// plan after its kernels have finished.
int mgk_density_counts_launch(mgk_ctx* ctx, const mgk_index* idx, const mgk_grid* g, int64_t row0, int64_t col0,
                              int64_t nr, int64_t nc, int slot, cudaStream_t s);
int mgk_density_plan_counted(mgk_ctx* ctx, const mgk_index* idx, const mgk_grid* g, int64_t row0, int64_t col0,
                             int64_t nr, int64_t nc, const float* d_mask, float* d_out, unsigned long long* d_evals,
                             int slot, mgk_dplan** out);
int mgk_density_launch_plan(mgk_ctx* ctx, mgk_dplan* plan, cudaStream_t s);
// The plan of rows/columns of a tile from per-block candidate counts in host
// memory (block-row major, ceil(nc / 128) per block row; e.g. a slice of one
// count of a larger tile whose block rows it shares); tables into `slot`.
int mgk_density_plan_from_counts(mgk_ctx* ctx, const mgk_index* idx, const mgk_grid* g, int64_t row0, int64_t col0,
                                 int64_t nr, int64_t nc, const int64_t* counts, const float* d_mask, float* d_out,
                                 unsigned long long* d_evals, int slot, mgk_dplan** out);
// Host view of the counts mgk_density_counts_launch wrote into `slot`.
const int64_t* mgk_density_counts_host(mgk_ctx* ctx, int slot);
// Copies a plan's work list from its staging slot to device memory on `s`
// now (mgk_density_launch_plan then skips that copy); the slot may be
// rewritten once this copy has run.
int mgk_density_stage(mgk_ctx* ctx, mgk_dplan* plan, cudaStream_t s);
// mgk_density_launch_plan with the merge of split blocks (if any) on
// s_merge, after the density on s (event ev); *merged_on_s_merge tells where
// the plan's last kernel went.
int mgk_density_launch_split(mgk_ctx* ctx, mgk_dplan* plan, cudaStream_t s, cudaStream_t s_merge, cudaEvent_t ev,
                             bool* merged_on_s_merge);
// The plan's density kernel sets *flag = 1 when its last CTA starts.
void mgk_density_set_tail_flag(mgk_dplan* plan, unsigned* flag);
// The plan's kernels read the tile's NoData mask as bits (device, 1 = valid,
// row r at byte r * stride, column c at bit c % 8 of byte c / 8) instead of floats.
void mgk_density_set_mask_bits(mgk_dplan* plan, const unsigned char* bits, int64_t stride);
int mgk_launch_mark_boundary(mgk_ctx* ctx, mgk_raster* r);
int mgk_raster_runs(mgk_ctx* ctx, mgk_raster* r);
int mgk_launch_dist2(mgk_ctx* ctx, mgk_points* p, mgk_raster* r, double cap);
int mgk_launch_edge_weights(mgk_ctx* ctx, int64_t n, const float* x, const float* y, const float* hpp,
                            float h, const double* dist2, const mgk_raster* r, float* ew_out,
                            unsigned long long* d_evals);
int mgk_launch_edge_weights_multi(mgk_ctx* ctx, int64_t n, const float* x, const float* y, const float* hpp,
                                  float hfix, const float* d_hgrid, int nh, const double* dist2,
                                  const mgk_raster* r, float* ew_out, int64_t ew_stride,
                                  unsigned long long* d_evals);

// Halo selection (index.cu): points of src inside a rectangle, input order.
// With dst == NULL: counts them into *count (d_scratch holds the per-tile
// offsets for the second call, mgk_points_select_scratch(n) unsigned).
int mgk_launch_points_select(mgk_ctx* ctx, const mgk_points* src, double xlo, double xhi, double ylo, double yhi,
                             unsigned* d_scratch, int64_t* count, mgk_points* dst);
int64_t mgk_points_select_scratch(int64_t n);

// Batched leave-one-out likelihood (loo.cu).
struct mgk_loo_batch;
int mgk_loo_batch_create(mgk_ctx* c, const mgk_points* p, const mgk_raster* r, float h_lo, float h_hi, int nh,
                         mgk_loo_batch** out);
int mgk_loo_batch_create_share(mgk_ctx* c, const mgk_points* p, const mgk_raster* r, float h_lo, float h_hi,
                               int nh, int part, int nparts, const float* ew_ext, int64_t ew_chunk,
                               mgk_loo_batch** out, bool replay = true);
int mgk_loo_batch_run(mgk_loo_batch* B, const float* hs, double* logl, int* best, int64_t* edge_evals,
                      int64_t* loo_evals);
void mgk_loo_batch_destroy(mgk_loo_batch* B);
