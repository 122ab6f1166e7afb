// Cell-binned point index, built on the GPU.
//
// Replaces the reference's CPU k-d tree and its flattened GPU copy
// (KDtree.cu:53-154, CUDA_KDtree.cu:26-102) and the per-tile host halo filter
// (ExtractSamplePointsCurTile, kde_cuda_kdtr_tiled.cu:4672-4747).  Points are
// put into square bins of side `side` over their bounding box and stored
// bin-major, so the points of any run of bins along a bin row are one
// contiguous range: a raster tile's candidates within 3h are a handful of
// ranges, one per bin row.
//
// The sort is a stable LSD radix sort of the bin id (digits of up to 9 bits,
// one kernel per digit), so the order inside a bin is the input order and
// every build is bitwise reproducible (the density sums are order-dependent
// in FP32).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "mgk_internal.cuh"

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kMaxDigits = 512;   // digits of up to 9 bits: 18-bit bin ids sort in two passes
constexpr int kMaxPasses = 4;     // 32-bit keys
// Looks at an earlier tile's state word before a digit is counted in its items instead.
#ifndef MGK_SORT_SPIN
#define MGK_SORT_SPIN (1ll << 24)
#endif
constexpr long long kSortSpin = MGK_SORT_SPIN;
// Bins up to which the gather fills the bin starts on its way instead of a
// kernel of searches (9 to 12 us of chained loads whatever the size).  A gap
// between two points can be all bins, which one warp then fills: 2^16 take it
// about as long as the searches.  Index builds on the way / by searches:
// 50,000 points in 7,600 bins 64 / 72 us, 200,000 in 2,000 70 / 83 us; a line at
// 2^12 or 2^18 is no faster.  With 2^19 points and more the build takes 120 us
// and up, and the sorted keys, which must outlive the gather's stores, stay in
// the record buffer instead of one of their own.
constexpr int64_t kFillBins = 1 << 16;
constexpr int kBuildLevels = 16;  // indexes built together
constexpr int kExtentCtas = 512;  // their words fit the context's mapped page

// The kernels of a build take up to N indexes of the same points (the levels of
// a bandwidth batch) in one launch: blockIdx.y is the index.
template <typename T, int N>
struct Jobs {
    T j[N];
};
struct KeyJob {
    double inv_side;
    int64_t nbx, nby;
    const MgkPt* pts;  // the records (Z-order keys), else null
    unsigned *keys, *hist;
};
struct SortJob {  // from (ka, indexes) through (kb, vb) and back
    unsigned *ka, *kb;
    int32_t *va, *vb;
    unsigned* scratch;
};
struct StartJob {
    const unsigned* keys;
    int64_t nbins;
    int32_t* start;
};
struct GatherJob {
    const int32_t* perm;
    MgkPt* out;
    int qexp;
    const unsigned* keys;  // the sorted keys, where the gather fills the bin starts, else null
    unsigned nbins;
    int32_t* start;
    int32_t* inv;  // the place of each point's record, or null
};

// The points' extent (and largest h): each CTA's ordered-integer minima and
// maxima (min x, min y, max x, max y, max h) into its words of mapped host
// memory, so that no copy goes through a copy engine.
__global__ void __launch_bounds__(256) k_extent(int64_t n, const float* __restrict__ x, const float* __restrict__ y,
                                                const float* __restrict__ h, unsigned* out) {
    __shared__ unsigned sh[8][5];
    unsigned v[5] = {0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned ox = mgk_f2ord(x[i]), oy = mgk_f2ord(y[i]);
        v[0] = min(v[0], ox);
        v[1] = min(v[1], oy);
        v[2] = max(v[2], ox);
        v[3] = max(v[3], oy);
        if (h) v[4] = max(v[4], mgk_f2ord(h[i]));
    }
#pragma unroll
    for (int k = 0; k < 5; k++) {
        v[k] = k < 2 ? __reduce_min_sync(0xffffffffu, v[k]) : __reduce_max_sync(0xffffffffu, v[k]);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5][k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        const int k = threadIdx.x;
        unsigned m = sh[0][k];
        for (int w = 1; w < 8; w++) m = k < 2 ? min(m, sh[w][k]) : max(m, sh[w][k]);
        out[blockIdx.x * 5 + k] = m;
    }
}

// Keys of a sort and the histograms of all their digits (pass p: bits
// [p db, (p + 1) db)) in one reading.
template <typename KeyOf>
__device__ __forceinline__ void keys_and_hist(int64_t n, const KeyOf& key_of, int db, int passes,
                                              unsigned* __restrict__ keys, unsigned* __restrict__ hist) {
    __shared__ unsigned sh[kMaxPasses * kMaxDigits];
    const int nd = 1 << db;
    for (int d = threadIdx.x; d < passes * nd; d += blockDim.x) sh[d] = 0;
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned k = key_of(i);
        keys[i] = k;
        for (int p = 0; p < passes; p++) atomicAdd(&sh[p * nd + ((k >> (p * db)) & (nd - 1))], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < passes * nd; d += blockDim.x)
        if (sh[d]) atomicAdd(&hist[d], sh[d]);
}

template <int N>
__global__ void __launch_bounds__(256) k_bin_keys(int64_t n, const float* __restrict__ x, const float* __restrict__ y,
                                                  double ox, double oy, int db, int passes,
                                                  const __grid_constant__ Jobs<KeyJob, N> J) {
    const KeyJob& B = J.j[N > 1 ? blockIdx.y : 0];
    const double inv_side = B.inv_side;
    const int64_t nbx = B.nbx, nby = B.nby;
    keys_and_hist(
        n,
        [&](int64_t i) {
            int64_t bx = (int64_t)floor(((double)x[i] - ox) * inv_side);
            int64_t by = (int64_t)floor(((double)y[i] - oy) * inv_side);
            bx = bx < 0 ? 0 : (bx >= nbx ? nbx - 1 : bx);
            by = by < 0 ? 0 : (by >= nby ? nby - 1 : by);
            return (unsigned)(by * nbx + bx);
        },
        db, passes, B.keys, B.hist);
}

// Exclusive scan of `len` counts in one CTA of 1024 threads (chunked).
__global__ void __launch_bounds__(1024) k_scan_exclusive(unsigned* __restrict__ data, int64_t len) {
    __shared__ unsigned long long part[1024];
    const int t = threadIdx.x;
    const int64_t chunk = (len + 1023) / 1024;
    const int64_t b = t * chunk, e = min(len, b + chunk);
    unsigned long long s = 0;
    for (int64_t i = b; i < e; i++) s += data[i];
    part[t] = s;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        unsigned long long v = t >= off ? part[t - off] : 0ull;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    unsigned long long run = t ? part[t - 1] : 0ull;
    for (int64_t i = b; i < e; i++) {
        unsigned v = data[i];
        data[i] = (unsigned)run;
        run += v;
    }
}

// Of the first n keys, those with digit d.
__device__ __forceinline__ unsigned count_digit(const unsigned* __restrict__ keys, int64_t n, int shift,
                                                unsigned mask, unsigned d) {
    unsigned c = 0;
#pragma unroll 1
    for (int64_t i = 0; i < n; i++) c += ((keys[i] >> shift) & mask) == d ? 1u : 0u;
    return c;
}

// One digit of the stable sort in one kernel.  Tiles of 256 IPT items are
// handed out in order by a counter; a tile ranks its items in registers (each
// warp its own run of 32 IPT, match_any per round), publishes its digit
// counts, and adds up those of the tiles before it, which are all running or
// done, from their published counts or sums (state in the top two bits of a
// word: 1 counts, 2 sums including all earlier tiles).  The wait for a word is
// bounded: after it the tile counts the earlier items itself, slowly, so the
// sort always ends and always sorts.  (Decoupled look back: Merrill and Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016.)  A pass
// reads and writes each item once; the earlier form (a histogram kernel, a scan
// of all tiles' counts in one CTA, a scatter in rounds of 256 items with five
// barriers each, tiles of 8,192) took 85 us a pass on 10^6 points and 29 us on
// 2,000, where one CTA did everything; this takes 36 and 6 us (an index build
// 289 -> 144 and 99 -> 54 us).  Before the first pass the values are the
// items' indexes.
template <int IPT, typename W, int N>
__global__ void __launch_bounds__(kSortThreads) k_radix_pass(int64_t n, int p, int passes, int db, size_t look_bytes,
                                                             const __grid_constant__ Jobs<SortJob, N> J) {
    const SortJob& B = J.j[N > 1 ? blockIdx.y : 0];
    const unsigned* __restrict__ keys_in = p & 1 ? B.kb : B.ka;
    const int32_t* __restrict__ vals_in = p == 0 ? nullptr : p & 1 ? B.vb : B.va;
    unsigned* __restrict__ keys_out = p & 1 ? B.ka : B.kb;
    int32_t* __restrict__ vals_out = p & 1 ? B.va : B.vb;
    const unsigned* __restrict__ hist = B.scratch + (p << db);
    unsigned* tick = B.scratch + (passes << db) + p;
    W* look = reinterpret_cast<W*>(reinterpret_cast<char*>(B.scratch + (passes << db) + 8) + p * look_bytes);
    const int shift = p * db;
    constexpr int kTop = sizeof(W) * 8 - 2;
    constexpr W kVal = ((W)1 << kTop) - 1;
    __shared__ unsigned cnt[kSortWarps][kMaxDigits];  // a warp's digit counts, then its offsets in the tile
    __shared__ unsigned base[kMaxDigits];             // items of smaller digits, then the tile's first place
    __shared__ unsigned wsum[kSortWarps];
    __shared__ unsigned s_tile;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int nd = 1 << db;
    if (t == 0) s_tile = atomicAdd(tick, 1u);
    for (int d = t; d < nd; d += kSortThreads)
        for (int w = 0; w < kSortWarps; w++) cnt[w][d] = 0;
    // exclusive scan of the digits' counts (one or two digits per thread)
    const int per = nd > kSortThreads ? 2 : 1;
    unsigned h0 = t * per < nd ? hist[t * per] : 0u, h1 = per == 2 ? hist[2 * t + 1] : 0u;
    unsigned sum = h0 + h1;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    if (lane == 31) wsum[wid] = sum;
    __syncthreads();
    for (int w = 0; w < wid; w++) sum += wsum[w];
    if (t * per < nd) {
        base[t * per] = sum - h0 - h1;
        if (per == 2) base[2 * t + 1] = sum - h1;
    }
    const unsigned tile = s_tile;
    const int64_t i0 = (int64_t)tile * (kSortThreads * IPT) + wid * (32 * IPT) + lane;
    unsigned key[IPT], rank[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) key[k] = i0 + 32 * k < n ? keys_in[i0 + 32 * k] : 0u;
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const bool valid = i0 + 32 * k < n;
        const unsigned d = valid ? (key[k] >> shift) & (nd - 1) : (unsigned)kMaxDigits;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned before = valid ? cnt[wid][d] : 0u;
        rank[k] = before + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (valid && (peers >> lane) == 1u) cnt[wid][d] = before + __popc(peers);  // the last of the peers
        __syncwarp();
    }
    __syncthreads();
    volatile W* lk = look;
    for (int d = t; d < nd; d += kSortThreads) {
        unsigned run = 0;
        for (int w = 0; w < kSortWarps; w++) {
            const unsigned c = cnt[w][d];
            cnt[w][d] = run;
            run += c;
        }
        lk[(size_t)tile * nd + d] = ((W)(tile ? 1 : 2) << kTop) | run;
        unsigned prev = 0;
        for (unsigned q = tile; q > 0;) {
            q--;
            W v = 0;
            long long spin = 0;
            while ((v = lk[(size_t)q * nd + d]) >> kTop == 0 && ++spin < kSortSpin) {
            }
            if (v >> kTop == 0) {
                prev += count_digit(keys_in, (int64_t)(q + 1) * (kSortThreads * IPT), shift, (unsigned)nd - 1u, (unsigned)d);
                break;
            }
            prev += (unsigned)(v & kVal);
            if (v >> kTop != 1) break;
        }
        if (tile) lk[(size_t)tile * nd + d] = ((W)2 << kTop) | (W)(prev + run);
        base[d] += prev;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const int64_t i = i0 + 32 * k;
        if (i >= n) continue;
        const unsigned d = (key[k] >> shift) & (nd - 1);
        const unsigned pos = base[d] + cnt[wid][d] + rank[k];
        keys_out[pos] = key[k];
        vals_out[pos] = vals_in ? vals_in[i] : (int32_t)i;
    }
}

// Passes and digit bits of a sort of `bits`-bit keys; its scratch words.
struct SortPlan {
    int passes, db, ipt;
    int64_t ntiles;
    bool wide;  // counts of 2^30 items and more: 64-bit state words
    size_t look_bytes() const { return (size_t)ntiles * ((size_t)1 << db) * (wide ? 8 : 4); }
    size_t bytes() const {  // [digit counts | tile counters | state words], zeroed before the keys
        return sizeof(unsigned) * (((size_t)passes << db) + 8) + (size_t)passes * look_bytes();
    }
};

// spare: the least scratch instead of the tiles that sort fastest.
SortPlan sort_plan(int64_t n, int bits, bool spare) {
    SortPlan P;
    bits = std::max(bits, 1);
    P.passes = (bits + 8) / 9;
    P.db = (bits + P.passes - 1) / P.passes;
    // Large tiles shorten the look back, small ones keep the SMs busy: 16, 4, 4
    // items a thread instead took 161 us for 10^6 points (144 with 16) and 4, 1
    // for 200,000 125 us (109 with 4).
    P.ipt = spare || n >= (1 << 19) ? 16 : n >= (1 << 16) ? 4 : 1;
    P.ntiles = (n + (int64_t)kSortThreads * P.ipt - 1) / ((int64_t)kSortThreads * P.ipt);
    P.wide = n >= (1ll << 30);
    return P;
}

// Sorts the keys in ka (values: indexes) with the histograms already in the
// scratch; the sorted keys and values end in kb, vb after an odd number of
// passes, else in ka, va.
template <int N>
void sort_passes(cudaStream_t s, const SortPlan& P, int64_t n, int nj, const Jobs<SortJob, N>& J) {
    const dim3 g((unsigned)P.ntiles, (unsigned)nj);
    for (int p = 0; p < P.passes; p++) {
        if (P.wide)
            k_radix_pass<16, unsigned long long, N><<<g, kSortThreads, 0, s>>>(n, p, P.passes, P.db, P.look_bytes(),
                                                                              J);
        else if (P.ipt == 16)
            k_radix_pass<16, unsigned, N><<<g, kSortThreads, 0, s>>>(n, p, P.passes, P.db, P.look_bytes(), J);
        else if (P.ipt == 4)
            k_radix_pass<4, unsigned, N><<<g, kSortThreads, 0, s>>>(n, p, P.passes, P.db, P.look_bytes(), J);
        else
            k_radix_pass<1, unsigned, N><<<g, kSortThreads, 0, s>>>(n, p, P.passes, P.db, P.look_bytes(), J);
    }
}

// start[b] = first sorted position whose key >= b  (b in [0, nbins]).  A warp
// takes STRETCHES x 32 bins: searches bound each stretch's positions, and
// where the bounds differ each bin is searched between them (empty stretches
// are plain stores; one thread per point filling the gap before its key took
// 58 us on 800,000 points in 7.5 million bins, where the gaps are long, this
// 36 us).  One stretch per warp where that leaves warps enough for the GPU
// (the searches are chains of loads), eight above 2^20 bins.
template <int STRETCHES, int N>
__global__ void __launch_bounds__(256) k_bin_starts(int64_t n, const __grid_constant__ Jobs<StartJob, N> J) {
    const StartJob& B = J.j[N > 1 ? blockIdx.y : 0];
    if (!B.start) return;  // the gather fills these
    const unsigned* __restrict__ keys = B.keys;
    const int64_t nbins = B.nbins;
    int32_t* __restrict__ start = B.start;
    const int lane = threadIdx.x & 31;
    const int64_t b0 = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * (32 * STRETCHES);
    if (b0 > nbins) return;
    auto first_at = [&](int64_t b, int64_t lo, int64_t hi) {  // first position in [lo, hi] with key >= b
        while (lo < hi) {
            const int64_t m = lo + ((hi - lo) >> 1);
            if ((int64_t)keys[m] >= b) hi = m;
            else lo = m + 1;
        }
        return lo;
    };
    // lanes 0..STRETCHES bound the stretches
    int64_t edge = 0;
    if (lane <= STRETCHES) edge = first_at(b0 + 32 * lane, 0, n);
    for (int k = 0; k < STRETCHES; k++) {
        const int64_t lo = __shfl_sync(0xffffffffu, edge, k), hi = __shfl_sync(0xffffffffu, edge, k + 1);
        const int64_t b = b0 + 32 * k + lane;
        if (b <= nbins) start[b] = (int32_t)first_at(b, lo, hi);
    }
}

// The starts of the bins after the key at i - 1, up to the key at i, are i
// (after the last key: n).  Gaps of more than four bins are filled by the warp.
__device__ __forceinline__ void fill_starts(int64_t n, int64_t i, const unsigned* __restrict__ keys, unsigned nbins,
                                            int32_t* __restrict__ start) {
    const int lane = threadIdx.x & 31;
    unsigned lo = 0, hi = 0;  // start[lo, hi) = i
    if (i <= n) {
        if (i > 0) lo = keys[i - 1] + 1;
        hi = (i < n ? keys[i] : nbins) + 1;
    }
    const bool wide = hi > lo + 4;
    if (!wide)
        for (unsigned b = lo; b < hi; b++) start[b] = (int32_t)i;
    for (unsigned m = __ballot_sync(0xffffffffu, wide); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const unsigned l = __shfl_sync(0xffffffffu, lo, src), h = __shfl_sync(0xffffffffu, hi, src);
        const int32_t at = (int32_t)(i - lane + src);
        for (unsigned b = l + lane; b < h; b += 32) start[b] = at;
    }
}

// A record's weight: w * e, divided by h^2 TWO_PI for per-point bandwidths
// (the per-point normalisation of the kernel).
__device__ __forceinline__ float record_wk(const float* __restrict__ w, const float* __restrict__ ew,
                                          const float* __restrict__ hpp, int32_t j) {
    float wk = (w ? w[j] : 1.0f) * (ew ? ew[j] : 1.0f);
    if (hpp) {
        const float hh = hpp[j] * hpp[j];
        wk = (float)((double)wk / ((double)hh * (double)MGK_TWO_PI_F));
    }
    return wk;
}

// The records' weights again, from the points' current edge weights.
__global__ void k_refresh_wk(int64_t n, const int32_t* __restrict__ perm, const float* __restrict__ w,
                             const float* __restrict__ ew, const float* __restrict__ hpp, MgkPt* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i].wk = record_wk(w, ew, hpp, perm[i]);
}

template <int N>
__global__ void k_gather(int64_t n, const float* __restrict__ x, const float* __restrict__ y,
                         const float* __restrict__ w, const float* __restrict__ ew, const float* __restrict__ hpp,
                         const __grid_constant__ Jobs<GatherJob, N> J) {
    const GatherJob& B = J.j[N > 1 ? blockIdx.y : 0];
    const int32_t* __restrict__ perm = B.perm;
    MgkPt* __restrict__ out = B.out;
    const int qexp = B.qexp;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (B.keys) fill_starts(n, i, B.keys, B.nbins, B.start);
    if (i >= n) return;
    const int32_t j = perm[i];
    if (B.inv) B.inv[j] = (int32_t)i;
    MgkPt r;
    mgk_qsplit(x[j], qexp, r.xh, r.xl);
    mgk_qsplit(y[j], qexp, r.yh, r.yl);
    r.wk = record_wk(w, ew, hpp, j);
    r.k2h = r.k2l = r.hh = 0.0f;
    if (hpp) {
        const float hh = hpp[j] * hpp[j];
        const double h2 = (double)hh;
        const double k2 = MGK_LOG2E / (2.0 * h2);
        r.k2h = (float)k2;
        r.k2l = (float)(k2 - (double)r.k2h);
        r.hh = hh;
    }
    out[i] = r;
}

// Z-order (Morton) key of the bin of each index record: bit-interleaved bin
// column and row (16 bits each), value = the record's position.
__device__ __forceinline__ unsigned spread16(unsigned v) {
    v &= 0xffffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}

template <int N>
__global__ void __launch_bounds__(256) k_morton_keys(int64_t n, double ox, double oy, int db, int passes,
                                                     const __grid_constant__ Jobs<KeyJob, N> J) {
    const KeyJob& B = J.j[N > 1 ? blockIdx.y : 0];
    const MgkPt* __restrict__ pts = B.pts;
    const double inv_side = B.inv_side;
    const int64_t nbx = B.nbx, nby = B.nby;
    keys_and_hist(
        n,
        [&](int64_t i) {
            const float4 p = *reinterpret_cast<const float4*>(pts + i);
            int64_t bx = (int64_t)floor(((double)(p.x + p.z) - ox) * inv_side);
            int64_t by = (int64_t)floor(((double)(p.y + p.w) - oy) * inv_side);
            bx = bx < 0 ? 0 : (bx >= nbx ? nbx - 1 : bx);
            by = by < 0 ? 0 : (by >= nby ? nby - 1 : by);
            return spread16((unsigned)bx) | (spread16((unsigned)by) << 1);
        },
        db, passes, B.keys, B.hist);
}

// Place along the Hilbert curve (Hilbert, 1891) of a point's cell in a 65,536 x
// 65,536 raster over the extent: quadrant by quadrant, each reflected and
// rotated as the curve's definition has it.
__global__ void __launch_bounds__(256) k_hilbert_keys(int64_t n, const float* __restrict__ x,
                                                      const float* __restrict__ y, double ox, double oy, double scale,
                                                      int db, int passes, unsigned* __restrict__ keys,
                                                      unsigned* __restrict__ hist) {
    keys_and_hist(
        n,
        [&](int64_t i) {
            unsigned u = (unsigned)fmin(fmax(((double)x[i] - ox) * scale, 0.0), 65535.0);
            unsigned v = (unsigned)fmin(fmax(((double)y[i] - oy) * scale, 0.0), 65535.0);
            unsigned d = 0;
            for (int b = 15; b >= 0; b--) {
                const unsigned ru = (u >> b) & 1u, rv = (v >> b) & 1u;
                d = (d << 2) | ((3u * ru) ^ rv);
                if (!rv) {
                    if (ru) {
                        u = ~u;
                        v = ~v;
                    }
                    const unsigned t = u;
                    u = v;
                    v = t;
                }
            }
            return d;
        },
        db, passes, keys, hist);
}

// ---- halo selection: the points inside a rectangle, in input order -------
constexpr int kSelThreads = 256;
constexpr int kSelRounds = 16;
constexpr int kSelTile = kSelThreads * kSelRounds;

struct SelRect {
    double xlo, xhi, ylo, yhi;
};

__device__ __forceinline__ bool sel_in(const SelRect& R, float x, float y) {
    const double dx = (double)x, dy = (double)y;
    return dx >= R.xlo && dx <= R.xhi && dy >= R.ylo && dy <= R.yhi;
}

// Kept points per tile of kSelTile points; counts[ntiles] = 0 (the scan's total slot).
__global__ void __launch_bounds__(kSelThreads) k_sel_count(int64_t n, const float* __restrict__ x,
                                                           const float* __restrict__ y, SelRect R, int ntiles,
                                                           unsigned* __restrict__ counts) {
    __shared__ unsigned s_c;
    if (threadIdx.x == 0) s_c = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSelTile;
    unsigned c = 0;
    for (int r = 0; r < kSelRounds; r++) {
        const int64_t i = base + (int64_t)r * kSelThreads + threadIdx.x;
        c += (i < n && sel_in(R, x[i], y[i])) ? 1u : 0u;
    }
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_c, c);
    __syncthreads();
    if (threadIdx.x == 0) {
        counts[blockIdx.x] = s_c;
        if (blockIdx.x == 0) counts[ntiles] = 0;
    }
}

// Stable scatter: round-major, thread-minor order is the input order; the
// rank of a kept point is its warp ballot rank plus the kept points of lower
// warps in the round and of earlier rounds.
__global__ void __launch_bounds__(kSelThreads) k_sel_scatter(
    int64_t n, const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ w,
    const float* __restrict__ h, SelRect R, const unsigned* __restrict__ offsets, float* __restrict__ ox,
    float* __restrict__ oy, float* __restrict__ ow, float* __restrict__ oh) {
    __shared__ unsigned s_w[kSelThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kSelTile;
    unsigned run = offsets[blockIdx.x];
    for (int r = 0; r < kSelRounds; r++) {
        const int64_t i = base + (int64_t)r * kSelThreads + threadIdx.x;
        const bool keep = i < n && sel_in(R, x[i], y[i]);
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) s_w[warp] = __popc(bal);
        __syncthreads();
        unsigned before = 0, total = 0;
        for (int k = 0; k < kSelThreads / 32; k++) {
            before += k < warp ? s_w[k] : 0u;
            total += s_w[k];
        }
        if (keep) {
            const unsigned o = run + before + __popc(bal & ((1u << lane) - 1u));
            ox[o] = x[i];
            oy[o] = y[i];
            if (ow) ow[o] = w[i];
            if (oh) oh[o] = h[i];
        }
        run += total;
        __syncthreads();  // s_w is rewritten next round
    }
}

}  // namespace

// The points of src inside [xlo, xhi] x [ylo, yhi] (input order) into dst,
// whose arrays the caller allocates after the count: first call with dst ==
// NULL returns the count in *count (one read back), then with dst.
int mgk_launch_points_select(mgk_ctx* ctx, const mgk_points* src, double xlo, double xhi, double ylo, double yhi,
                             unsigned* d_scratch, int64_t* count, mgk_points* dst) {
    const int64_t n = src->n;
    const int ntiles = (int)((n + kSelTile - 1) / kSelTile);
    const SelRect R{xlo, xhi, ylo, yhi};
    cudaStream_t s = ctx->stream;
    if (!dst) {
        if (n == 0) {
            *count = 0;
            return MGK_OK;
        }
        k_sel_count<<<ntiles, kSelThreads, 0, s>>>(n, src->x, src->y, R, ntiles, d_scratch);
        k_scan_exclusive<<<1, 1024, 0, s>>>(d_scratch, ntiles + 1);
        MGK_CHECK_LAUNCH(ctx, "points select count");
        MGK_COUNT_LAUNCH(ctx, 2);
        unsigned tot = 0;
        MGK_CHECK_CUDA(ctx, cudaMemcpyAsync(&tot, d_scratch + ntiles, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        MGK_CHECK_CUDA(ctx, cudaStreamSynchronize(s));
        *count = (int64_t)tot;
        return MGK_OK;
    }
    if (n == 0 || dst->n == 0) return MGK_OK;
    k_sel_scatter<<<ntiles, kSelThreads, 0, s>>>(n, src->x, src->y, src->w, src->h, R, d_scratch, dst->x, dst->y,
                                                 src->w ? dst->w : nullptr, src->h ? dst->h : nullptr);
    MGK_CHECK_LAUNCH(ctx, "points select scatter");
    MGK_COUNT_LAUNCH(ctx, 1);
    return MGK_OK;
}

// CTAs of a key kernel.
static unsigned key_grid(const mgk_ctx* ctx, int64_t n) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 4 * (int64_t)ctx->sm_count));
}

int64_t mgk_points_select_scratch(int64_t n) { return (n + kSelTile - 1) / kSelTile + 1; }

// One index's sort scratch: two key buffers, a value buffer, and the zeroed
// digit counts and state words.
struct SortBuf {
    unsigned *k0, *k1;
    int32_t* v0;
    unsigned* scr;
};

static size_t up256(size_t v) { return (v + 255) / 256 * 256; }

static SortPlan bin_plan(int64_t n, int64_t nbins, bool spare = false) {
    int bits = 0;
    while (bits < 32 && ((uint64_t)(nbins - 1) >> bits) != 0) bits++;
    return sort_plan(n, bits, spare);
}

static SortPlan zorder_plan(int64_t n, int64_t nbx, int64_t nby, bool spare = false) {
    const uint64_t maxb = (uint64_t)std::max(nbx, nby) - 1;
    int bits = 0;
    while (bits < 16 && (maxb >> bits) != 0) bits++;
    return sort_plan(n, 2 * bits, spare);
}

// The records, their permutation and the bin starts of nj indexes of the same
// points, sorted by plan P (digits enough for the largest bin grid).  own: the
// scratch is not the record buffer, so the sorted keys outlive the gather's
// first stores.
template <int N>
static cudaError_t enqueue_build(mgk_ctx* ctx, const mgk_points* pts, bool varh, int nj, mgk_index* const* idx,
                                 const SortBuf* buf, bool own, const SortPlan& P,
                                 int32_t* inv) {
    const int64_t n = pts->n;
    cudaStream_t s = ctx->stream;
    const bool odd = P.passes & 1;  // the values end in perm
    int64_t nbins = 0;
    bool search = false;  // for some index's bin starts
    Jobs<KeyJob, N> K{};
    Jobs<SortJob, N> S{};
    Jobs<StartJob, N> T{};
    Jobs<GatherJob, N> G{};
    for (int j = 0; j < nj; j++) {
        const mgk_index* I = idx[j];
        const SortBuf& b = buf[j];
        nbins = std::max(nbins, I->nbx * I->nby);
        K.j[j] = KeyJob{1.0 / I->side, I->nbx, I->nby, nullptr, b.k0, b.scr};
        S.j[j] = SortJob{b.k0, b.k1, odd ? b.v0 : I->perm, odd ? I->perm : b.v0, b.scr};
        T.j[j] = StartJob{odd ? b.k1 : b.k0, I->nbx * I->nby, I->bin_start};
        G.j[j] = GatherJob{I->perm, I->pts, I->qexp, nullptr, 0u, nullptr, inv};
        if (own && T.j[j].nbins <= kFillBins) {
            G.j[j].keys = T.j[j].keys;
            G.j[j].nbins = (unsigned)T.j[j].nbins;
            std::swap(G.j[j].start, T.j[j].start);
        } else {
            search = true;
        }
    }
    const unsigned ny = (unsigned)nj;
    k_bin_keys<N><<<dim3(key_grid(ctx, n), ny), 256, 0, s>>>(n, pts->x, pts->y, idx[0]->ox, idx[0]->oy, P.db, P.passes,
                                                             K);
    sort_passes<N>(s, P, n, nj, S);
    if (search && nbins < (1 << 20))
        k_bin_starts<1, N><<<dim3((unsigned)(nbins / 256 + 1), ny), 256, 0, s>>>(n, T);
    else if (search)
        k_bin_starts<8, N><<<dim3((unsigned)(nbins / 2048 + 1), ny), 256, 0, s>>>(n, T);
    k_gather<N><<<dim3((unsigned)(n / 256 + 1), ny), 256, 0, s>>>(  // a thread past the last record ends the starts
        n, pts->x, pts->y, pts->w, pts->has_ew ? pts->ew : nullptr, varh ? pts->h : nullptr, G);
    MGK_COUNT_LAUNCH(ctx, (search ? 3 : 2) + P.passes);
    return cudaGetLastError();
}

// Positions of the records of nj indexes in Z-order of their bins (stable:
// records of one bin keep their order).  Consecutive runs of this order are
// compact in both directions, unlike runs of the row-major record order.
template <int N>
static cudaError_t enqueue_zorder(mgk_ctx* ctx, int nj, mgk_index* const* idx, int32_t* const* order,
                                  const SortBuf* buf, const SortPlan& P) {
    const int64_t n = idx[0]->n;
    const bool odd = P.passes & 1;  // the values end in order
    Jobs<KeyJob, N> K{};
    Jobs<SortJob, N> S{};
    for (int j = 0; j < nj; j++) {
        const mgk_index* I = idx[j];
        const SortBuf& b = buf[j];
        K.j[j] = KeyJob{1.0 / I->side, I->nbx, I->nby, I->pts, b.k0, b.scr};
        S.j[j] = SortJob{b.k0, b.k1, odd ? b.v0 : order[j], odd ? order[j] : b.v0, b.scr};
    }
    k_morton_keys<N><<<dim3(key_grid(ctx, n), (unsigned)nj), 256, 0, ctx->stream>>>(n, idx[0]->ox, idx[0]->oy, P.db,
                                                                                    P.passes, K);
    sort_passes<N>(ctx->stream, P, n, nj, S);
    MGK_COUNT_LAUNCH(ctx, 1 + P.passes);
    return cudaGetLastError();
}

// Runs enqueue(scratch, plan) with a sort's zeroed scratch for n items: in one
// block, or without the memory for that by the plan of the least scratch in
// blocks of their own.  plan_of(spare): the sort's plan.
template <typename PlanOf, typename Enqueue>
static int with_sort_buf(mgk_ctx* ctx, int64_t n, const PlanOf& plan_of, const char* what, const Enqueue& enqueue) {
    SortPlan P = plan_of(false);
    const size_t b_buf = up256(sizeof(unsigned) * (size_t)n), b_one = 3 * b_buf + P.bytes();
    void* blk[4] = {};
    size_t b_blk[4] = {b_one, b_buf, b_buf, b_buf};
    SortBuf b{};
    int st;
    if ((st = mgk_alloc(ctx, &blk[0], b_one)) == MGK_OK) {
        char* base = static_cast<char*>(blk[0]);
        b = SortBuf{(unsigned*)base, (unsigned*)(base + b_buf), (int32_t*)(base + 2 * b_buf),
                    (unsigned*)(base + 3 * b_buf)};
    } else {
        P = plan_of(true);
        b_blk[0] = P.bytes();
        st = MGK_OK;
        for (int i = 0; i < 4 && st == MGK_OK; i++) st = mgk_alloc(ctx, &blk[i], b_blk[i]);
        b = SortBuf{(unsigned*)blk[1], (unsigned*)blk[2], (int32_t*)blk[3], (unsigned*)blk[0]};
    }
    cudaError_t e = cudaSuccess;
    if (st == MGK_OK) e = cudaMemsetAsync(b.scr, 0, P.bytes(), ctx->stream);
    if (st == MGK_OK && e == cudaSuccess) e = enqueue(b, P);
    // back to the context's pool; later users are ordered after these kernels on the same stream
    for (int i = 0; i < 4; i++) mgk_free(ctx, blk[i], b_blk[i]);
    if (e != cudaSuccess) return mgk_cuda_fail(ctx, e, what);
    return st;
}

// Z-order of one index's records.
static int index_zorder(mgk_ctx* ctx, mgk_index* idx, int32_t* d_order) {
    return with_sort_buf(
        ctx, idx->n, [&](bool spare) { return zorder_plan(idx->n, idx->nbx, idx->nby, spare); }, "index_zorder",
        [&](const SortBuf& b, const SortPlan& P) { return enqueue_zorder<1>(ctx, 1, &idx, &d_order, &b, P); });
}

int mgk_points_curve_order(mgk_ctx* ctx, const mgk_points* pts, const mgk_extent& extent, int32_t* d_order) {
    const int64_t n = pts->n;
    if (n == 0) return MGK_OK;
    const double ext = std::max(extent.xmax - extent.xmin, extent.ymax - extent.ymin);
    return with_sort_buf(
        ctx, n, [&](bool spare) { return sort_plan(n, 32, spare); }, "points_curve_order",
        [&](const SortBuf& b, const SortPlan& P) {
            const bool odd = P.passes & 1;  // the values end in d_order
            Jobs<SortJob, 1> S{};
            S.j[0] = SortJob{b.k0, b.k1, odd ? b.v0 : d_order, odd ? d_order : b.v0, b.scr};
            k_hilbert_keys<<<key_grid(ctx, n), 256, 0, ctx->stream>>>(n, pts->x, pts->y, extent.xmin, extent.ymin,
                                                                      ext > 0.0 ? 65536.0 / ext : 0.0, P.db, P.passes,
                                                                      b.k0, b.scr);
            sort_passes<1>(ctx->stream, P, n, 1, S);
            MGK_COUNT_LAUNCH(ctx, 1 + P.passes);
            return cudaGetLastError();
        });
}

int mgk_index_refresh_weights(mgk_ctx* ctx, mgk_index* idx, const mgk_points* pts) {
    if (!idx || !pts || idx->n != pts->n) return mgk_fail(ctx, MGK_ERR_INVALID, "index_refresh_weights: bad arguments");
    if (idx->n == 0) return MGK_OK;
    k_refresh_wk<<<(unsigned)((idx->n + 255) / 256), 256, 0, ctx->stream>>>(
        idx->n, idx->perm, pts->w, pts->has_ew ? pts->ew : nullptr, idx->varh ? pts->h : nullptr, idx->pts);
    MGK_CHECK_LAUNCH(ctx, "k_refresh_wk");
    MGK_COUNT_LAUNCH(ctx, 1);
    return MGK_OK;
}

// Extent of the points and, with want_h, their largest h (waits for the
// stream).  No points: the unit square.
int mgk_points_extent(mgk_ctx* ctx, const mgk_points* pts, bool want_h, mgk_extent* out) {
    *out = mgk_extent{};
    if (pts->n <= 0) return MGK_OK;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(kExtentCtas, (pts->n + 1023) / 1024));
    k_extent<<<blocks, 256, 0, ctx->stream>>>(pts->n, pts->x, pts->y, want_h ? pts->h : nullptr, ctx->d_map + 64);
    MGK_CHECK_LAUNCH(ctx, "k_extent");
    MGK_COUNT_LAUNCH(ctx, 1);
    MGK_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const volatile unsigned* m = ctx->h_map + 64;
    unsigned v[5] = {0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    for (int b = 0; b < blocks; b++)
        for (int k = 0; k < 5; k++) {
            const unsigned u = m[5 * b + k];
            v[k] = k < 2 ? std::min(v[k], u) : std::max(v[k], u);
        }
    out->xmin = mgk_ord2f(v[0]);
    out->ymin = mgk_ord2f(v[1]);
    out->xmax = mgk_ord2f(v[2]);
    out->ymax = mgk_ord2f(v[3]);
    if (want_h) out->hmax = mgk_ord2f(v[4]);
    return MGK_OK;
}

// An index's numbers and its arrays, without the kernels that fill them.
// extent: the points' (with per-point h: their largest h too) if known, else null.
static int index_plan(mgk_ctx* ctx, const mgk_points* pts, float h, float bin_size, const mgk_extent* extent,
                      mgk_index* idx) {
    const int64_t n = pts->n;
    idx->ctx = ctx;
    idx->n = n;
    idx->varh = (h <= 0.0f);
    if (idx->varh && !pts->h) return mgk_fail(ctx, MGK_ERR_INVALID, "index_build: h <= 0 but the points carry no per-point h");
    if (n >= (int64_t)INT32_MAX) return mgk_fail(ctx, MGK_ERR_INVALID, "index_build: too many points");
    int st;
    mgk_extent ext_own;
    if (!extent) {
        if ((st = mgk_points_extent(ctx, pts, idx->varh, &ext_own))) return st;
        extent = &ext_own;
    }
    const double xmin = extent->xmin, ymin = extent->ymin, xmax = extent->xmax, ymax = extent->ymax;
    float hmax = h;
    if (idx->varh) hmax = n > 0 ? extent->hmax : 1.0f;
    if (!(hmax > 0.0f) || !std::isfinite(hmax)) return mgk_fail(ctx, MGK_ERR_INVALID, "index_build: bandwidths must be positive and finite");
    idx->h = idx->varh ? 0.0f : h;
    idx->h2 = mgk_h2(hmax);
    idx->cut_d2 = MGK_CUT * idx->h2;
    idx->k2 = MGK_LOG2E / (2.0 * idx->h2);
    idx->k0 = 1.0 / (idx->h2 * (double)MGK_TWO_PI_F);
    // 3h plus a margin: 9 h^2 is formed from the float square, which may
    // exceed h^2 by a relative 2^-24
    idx->reach = 3.0 * (double)hmax * (1.0 + 1e-6);
    double side = bin_size > 0.0f ? (double)bin_size : (double)ctx->bin_factor * (double)hmax;
    const double ext = std::max(xmax - xmin, ymax - ymin);
    side = std::max(side, ext / 4096.0);
    if (!(side > 0.0)) side = 1.0;
    idx->side = side;
    idx->ox = xmin;
    idx->oy = ymin;
    idx->nbx = (int64_t)std::floor((xmax - xmin) / side) + 1;
    idx->nby = (int64_t)std::floor((ymax - ymin) / side) + 1;
    const int64_t nbins = idx->nbx * idx->nby;
    // coordinate quantum: every coordinate within 3h (+ a bin) of a point is
    // below 2^(22 - qexp) in magnitude, so hi parts are exact floats and
    // differences of hi parts within the cutoff are exact
    const double maxabs = std::max(std::max(std::fabs(xmin), std::fabs(xmax)),
                                   std::max(std::fabs(ymin), std::fabs(ymax))) + 4.0 * idx->reach + 2.0 * side + 1.0;
    idx->qexp = 22 - (int)std::ceil(std::log2(maxabs));

    // allocations (persistent)
    const size_t b_start = sizeof(int32_t) * (size_t)(nbins + 1);
    const size_t b_pts = sizeof(MgkPt) * (size_t)std::max<int64_t>(n, 1);
    const size_t b_perm = sizeof(int32_t) * (size_t)std::max<int64_t>(n, 1);
    if ((st = mgk_alloc(ctx, (void**)&idx->bin_start, b_start))) return st;
    if ((st = mgk_alloc(ctx, (void**)&idx->pts, b_pts))) return st;
    if ((st = mgk_alloc(ctx, (void**)&idx->perm, b_perm))) return st;
    idx->bytes = b_start + b_pts + b_perm;
    return MGK_OK;
}

// Fills a planned index.
static int index_fill(mgk_ctx* ctx, const mgk_points* pts, mgk_index* idx, int32_t* inv = nullptr) {
    const int64_t n = pts->n, nbins = idx->nbx * idx->nby;
    cudaStream_t s = ctx->stream;
    if (n == 0) {
        MGK_CHECK_CUDA(ctx, cudaMemsetAsync(idx->bin_start, 0, sizeof(int32_t) * (size_t)(nbins + 1), s));
        return MGK_OK;
    }
    // The sort's scratch lies in the record buffer, which the gather fills
    // last, or, where the gather fills the bin starts or the record buffer is
    // too small, in a buffer of its own.  Without the memory for one, the plan of
    // the least scratch, which fits the record buffer from about 500 points.
    SortPlan P = bin_plan(n, nbins);
    const size_t b_buf = up256(sizeof(unsigned) * (size_t)n), room = sizeof(MgkPt) * (size_t)n;
    size_t need = 3 * b_buf + P.bytes();
    char* base = reinterpret_cast<char*>(idx->pts);
    void* own = nullptr;
    int st;
    if ((need > room || (nbins <= kFillBins && n < (1 << 19))) && mgk_alloc(ctx, &own, need) && need > room) {
        P = bin_plan(n, nbins, true);
        need = 3 * b_buf + P.bytes();
        if (need > room && (st = mgk_alloc(ctx, &own, need))) return st;
    }
    if (own) base = static_cast<char*>(own);
    const SortBuf b{(unsigned*)base, (unsigned*)(base + b_buf), (int32_t*)(base + 2 * b_buf),
                    (unsigned*)(base + 3 * b_buf)};
    cudaError_t e = cudaMemsetAsync(b.scr, 0, P.bytes(), s);
    if (e == cudaSuccess) e = enqueue_build<1>(ctx, pts, idx->varh, 1, &idx, &b, own != nullptr, P, inv);
    if (own) mgk_free(ctx, own, need);  // later users are ordered after these kernels on the same stream
    if (e != cudaSuccess) return mgk_cuda_fail(ctx, e, "index build");
    return MGK_OK;
}

int mgk_launch_index_build(mgk_ctx* ctx, const mgk_points* pts, float h, float bin_size, const mgk_extent* extent,
                           mgk_index* idx, int32_t* inv) {
    const int st = index_plan(ctx, pts, h, bin_size, extent, idx);
    return st ? st : index_fill(ctx, pts, idx, inv);
}

// The indexes of a bandwidth batch: bin sides side0 2^l for l < nlev, up to and
// including the first whose side the bin-count limit raised to the one before,
// each with the Z-order of its records.  All levels go through each kernel
// together: one level's kernels on 2,000 points are 8 CTAs and 3 to 8 us each,
// mostly launch and the chain of a tile's loads, so six levels one after the
// other took 210 us of the device in 42 launches.  Together they are 9
// launches: 16 bandwidths scored on 2,000 points 500 -> 281 us, a golden-section
// search on 20,000 points (seven levels) 3.91 -> 3.56 ms.
// From 2^19 points a level fills the GPU by itself, and the levels go one
// after the other, as they do without the memory for all levels' scratch.
int mgk_index_build_levels(mgk_ctx* ctx, const mgk_points* pts, float h, double side0, int nlev,
                           const mgk_extent* extent, std::vector<mgk_index*>* lev, std::vector<int32_t*>* order) {
    const int64_t n = pts->n;
    int st;
    SortPlan P{}, Z{};
    size_t nl = 0;
    for (int l = 0; l < nlev; l++) {
        mgk_index* I = new (std::nothrow) mgk_index();
        if (!I) return mgk_fail(ctx, MGK_ERR_INVALID, "index levels: out of host memory");
        if ((st = index_plan(ctx, pts, h, (float)std::ldexp(side0, l), extent, I))) {
            mgk_index_destroy(I);
            return st;
        }
        lev->push_back(I);
        int32_t* q = nullptr;
        if ((st = mgk_alloc(ctx, (void**)&q, sizeof(int32_t) * (size_t)std::max<int64_t>(n, 1)))) return st;
        order->push_back(q);
        nl++;
        if (l == 0) {  // the finest level has the most bins
            P = bin_plan(n, I->nbx * I->nby);
            Z = zorder_plan(n, I->nbx, I->nby);
        } else if (I->side <= (*lev)[l - 1]->side) {
            break;
        }
    }
    const size_t zp = up256(P.bytes()), zz = up256(Z.bytes()), zero = nl * (zp + zz);
    const size_t b_buf = up256(sizeof(unsigned) * (size_t)n), need = zero + nl * 3 * b_buf;
    char* base = nullptr;
    if (n == 0 || n >= (1 << 19) || nl == 1 || nl > kBuildLevels || mgk_alloc(ctx, (void**)&base, need)) {
        for (size_t l = 0; l < nl; l++) {
            if ((st = index_fill(ctx, pts, (*lev)[l]))) return st;
            if (n > 0 && (st = index_zorder(ctx, (*lev)[l], (*order)[l]))) return st;
        }
        return MGK_OK;
    }
    SortBuf bp[kBuildLevels], bz[kBuildLevels];
    for (size_t l = 0; l < nl; l++) {
        char* keys = base + zero + l * 3 * b_buf;
        bp[l] = SortBuf{(unsigned*)keys, (unsigned*)(keys + b_buf), (int32_t*)(keys + 2 * b_buf),
                        (unsigned*)(base + l * zp)};
        bz[l] = bp[l];
        bz[l].scr = (unsigned*)(base + nl * zp + l * zz);
    }
    cudaError_t e = cudaMemsetAsync(base, 0, zero, ctx->stream);
    if (e == cudaSuccess) e = enqueue_build<kBuildLevels>(ctx, pts, false, (int)nl, lev->data(), bp, true, P, nullptr);
    if (e == cudaSuccess) e = enqueue_zorder<kBuildLevels>(ctx, (int)nl, lev->data(), order->data(), bz, Z);
    mgk_free(ctx, base, need);  // later users are ordered after these kernels on the same stream
    if (e != cudaSuccess) return mgk_cuda_fail(ctx, e, "index levels");
    return MGK_OK;
}
