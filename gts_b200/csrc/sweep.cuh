// sweep.cuh -- what the row sweep (sweep.cu), the string sweep (sweep_edit.cu)
// and the fast form's small batches (fast_small.cu) share.
#pragma once
#include <cfloat>
#include <climits>
#include "search.cuh"

namespace gts {

constexpr int kSwCap = 2048;           // candidates listed per query
constexpr float kSwTiny = 1e-36f;      // squares below this may have lost bits to underflow

struct SweepArgs {
    SearchArgs a;
    int q0, nq, ntiles, Qp, ld;         // the run's queries a.qids[q0 ..], padded count, query row stride
    int tq;                             // queries per tile (row lists, ring bounds)
    int ncut, nanc;
    const int2 *cut;                    // (node, first object): pieces of at most kCutSize objects
    const int *anc, *anc_idx;
    const float *tnorm;                 // angle: norms of the rows in tree order
    int *key, *order;                   // tree position of the query; sorted order -> query of the run
    int *bq;                            // sorted slot -> query of the batch (-1: padding)
    float *seed;                        // per query of the run: bound on the k-th distance (kNN)
    float *qrow;                        // [Qp][ld] sorted query rows, zero padded
    float *R, *vthr, *vlow, *qnorm;     // per sorted query: radius, value thresholds
    int *self;                          // its tree position when it is an object (-1)
    float *dlo, *dhi;                   // [nanc][Qp] pivot distance bounds
    int *nrows, *rowpos;                // per tile: rows to look at, their positions [ntiles][num]
    int *ccnt, *cpos;                   // candidate lists [Qp][cap]
    float *cv;
    int *cnt, *cnt2;                    // range: certain counts per sorted query
    int *ctr;                           // [0] item counter, [1] queries left over, [2] of them (strings) for a full list
    int4 *left;                         // queries whose list overflowed: (query, 0, 0, 0) for the traversal
    float *left_R;                      // kNN: and a bound on their k-th distance, from the list
    const int4 *again;                  // kNN, a later round: the run's queries and bounds come from
    const float *again_R;               //   again[q0 ..], again_R[q0 ..]
    int cap;                            // candidates listed per query
    int sample;                         // look at every sample-th row only (1: all)
    const uint4 *lens_ok;               // strings: per tile a mask of the lengths some query can match (nullable)
};

// Upper / lower bound on the distance from a filter value, as value_bounds_f,
// with the squares that underflow may have cut allowed for.
__device__ __forceinline__ float sw_hi(int metric, int dim, float v)
{
    float lo, hi;
    value_bounds_f(metric, dim, metric == kL2 ? v + kSwTiny : v, lo, hi);
    return hi;
}
__device__ __forceinline__ float sw_lo(int metric, int dim, float v)
{
    float lo, hi;
    value_bounds_f(metric, dim, metric == kL2 ? fmaxf(v - kSwTiny, 0.f) : v, lo, hi);
    return lo;
}

// k-th smallest (k >= 1) of n non-negative floats given as bits in keys: four
// passes over their bytes.  All threads of the CTA call it and get the bits.
__device__ __forceinline__ uint32_t cta_kth(const uint32_t *keys, int n, int k, int *hist)
{
    __shared__ uint32_t s_prefix;
    __shared__ int s_rank;
    uint32_t prefix = 0;
    int rank = k;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        const uint32_t mask = shift == 24 ? 0u : 0xffffffffu << (shift + 8);
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            if ((keys[i] & mask) == prefix) atomicAdd(&hist[(keys[i] >> shift) & 255], 1);
        __syncthreads();
        if (threadIdx.x < 32) {
            int c[8], sum = 0;
#pragma unroll
            for (int u = 0; u < 8; u++) sum += c[u] = hist[threadIdx.x * 8 + u];
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += y;
            }
            int run = incl - sum;
            if (run < rank && rank <= incl)
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    if (run < rank && rank <= run + c[u]) {
                        s_prefix = prefix | ((uint32_t)(threadIdx.x * 8 + u) << shift);
                        s_rank = rank - run;
                    }
                    run += c[u];
                }
        }
        __syncthreads();
        prefix = s_prefix;
        rank = s_rank;
        __syncthreads();
    }
    return prefix;
}

constexpr int kSwBatch = 8;   // candidates a warp evaluates side by side

// The reference's kNN value (F64 accumulation, dist_row_f64) of up to
// kSwBatch rows against the query, row c's on lane c: the lanes make the terms
// of 32 dimensions of each row (coalesced), then lane c adds row c's in order.
//
// L2 terms: the reference's pow(e, 2) is within 2 ulp of the square, which is
// exact in FP64 for a float e and costs a multiplication (pow: 0.5 per clock
// and SM, which made it most of these kernels' time).  POW = false adds the
// squares, and the caller checks that the sums are clear of everything they
// decide (l2_margin).
template <bool POW>
__device__ __forceinline__ double exact_batch(int metric, int dim, const float *const (&row)[kSwBatch], int n,
                                              const float *q, double (*ts)[33], int lane)
{
    double r = 0.0;
    float x[kSwBatch], y = lane < dim ? q[lane] : 0.f;
#pragma unroll
    for (int c = 0; c < kSwBatch; c++) x[c] = c < n && lane < dim ? __ldg(row[c] + lane) : 0.f;
    for (int c0 = 0; c0 < dim; c0 += 32) {
#pragma unroll
        for (int c = 0; c < kSwBatch; c++)
            if (c < n) {
                const float e = x[c] - y;
                ts[c][lane] = metric != kL2 ? (double)fabsf(e) : (POW ? pow(e, 2) : (double)e * (double)e);
            }
        // the next 32 dimensions are on their way while lane c adds these
        const int j = c0 + 32 + lane;
        y = j < dim ? q[j] : 0.f;
#pragma unroll
        for (int c = 0; c < kSwBatch; c++) x[c] = c < n && j < dim ? __ldg(row[c] + j) : 0.f;
        __syncwarp();
        if (lane < n) {
            const int m = min(32, dim - c0);
            const double *e = ts[lane];
            if (metric == kLinf) {
                for (int u = 0; u < m; u++)
                    if (e[u] > r) r = e[u];
            } else {
#pragma unroll 8
                for (int u = 0; u < m; u++) r += e[u];
            }
        }
        __syncwarp();
    }
    return metric == kL2 ? pow(r, 0.5) : r;
}

// The reference's range value (F32 accumulation, dist_row_f32) of up to NB
// rows at positions pos (lane c's row: rows + pos * ld) against the query, on
// lane c.  The sum is a chain of some 25 instructions a term, so as many
// lanes as there are rows walk theirs side by side.
template <int NB>
__device__ __forceinline__ float range_batch(int metric, int dim, const float *rows, size_t ld, int pos, int n,
                                             const float *q, float (*ts)[33], int lane)
{
    float r = 0.f, x[NB], y = lane < dim ? q[lane] : 0.f;
    const float *row = rows + (size_t)pos * ld;
    auto load = [&](int c0) {
#pragma unroll
        for (int c = 0; c < NB; c++) {
            const float *p = reinterpret_cast<const float *>(
                __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(row), c < n ? c : n - 1));
            x[c] = c0 + lane < dim ? __ldg(p + c0 + lane) : 0.f;
        }
    };
    load(0);
    for (int c0 = 0; c0 < dim; c0 += 32) {
#pragma unroll
        for (int c = 0; c < NB; c++) ts[c][lane] = x[c] - y;
        // the next 32 dimensions are on their way while the lanes add these
        if (c0 + 32 < dim) {
            y = c0 + 32 + lane < dim ? q[c0 + 32 + lane] : 0.f;
            load(c0 + 32);
        }
        __syncwarp();
        if (lane < n) {
            const int m = min(32, dim - c0);
            const float *e = ts[lane];
            if (metric == kL2) {
#pragma unroll 4
                for (int u = 0; u < m; u++) r = add_square(r, e[u]);
            } else if (metric == kL1) {
                for (int u = 0; u < m; u++) r += fabsf(e[u]);
            } else {
                for (int u = 0; u < m; u++) {
                    const float v = fabsf(e[u]);
                    if (v > r) r = v;
                }
            }
        }
        __syncwarp();
    }
    if (metric == kL2) r = pow(r, 0.5);
    return r;
}

// Relative distance within which two L2 values summed from exact squares may
// differ from the reference's: 2 ulp per term and one rounding per addition,
// halved by the root, with a factor above 2 to spare (1e-13 at dim 320).
__device__ __forceinline__ double l2_margin(int dim) { return 3.2e-16 * (double)(dim + 8); }

// Whether an L2 value d summed from exact squares may round to another float
// than the reference's.
__device__ __forceinline__ bool rounds_riskily(double d, double margin)
{
    if (d == 0.0) return false;   // all terms zero: exact
    const float f = __double2float_rn(d);
    const double fd = f, dl = d * margin;
    const double hi = 0.5 * (fd + (double)__int_as_float(__float_as_int(f) + 1));
    const double lo = 0.5 * (fd + (double)__int_as_float(__float_as_int(f) - 1));
    return !(f > 0.f && d - dl > lo && d + dl < hi);
}

struct FinalSmem {
    double d[kSwCap];
    int id[kSwCap];
    uint32_t key[kSwCap];
    int pos[kSwCap];
    double ts[4][kSwBatch][33];
    int hist[256];
    int n, risk;
};

// Ascending (distance, id) order of the first n entries.
__device__ __forceinline__ void sort_hits(FinalSmem &s, int n)
{
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    for (int i = n + threadIdx.x; i < p2; i += blockDim.x) {
        s.d[i] = DBL_MAX;
        s.id[i] = INT_MAX;
    }
    __syncthreads();
    for (int size = 2; size <= p2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < p2 / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const bool up = (lo & size) == 0;
                const double dl = s.d[lo], dh = s.d[hi];
                const int il = s.id[lo], ih = s.id[hi];
                if (((dl > dh) || (dl == dh && il > ih)) == up) {
                    s.d[lo] = dh;
                    s.d[hi] = dl;
                    s.id[lo] = ih;
                    s.id[hi] = il;
                }
            }
            __syncthreads();
        }
}

// kNN values of the n rows at f.pos (slots of `rows`, stride ld; ids of the
// slots in ids; the query's own slot `self` at 0) into f.d / f.id, in
// (distance, id) order.  128 threads.  L2 values come from exact squares
// unless that could change a float or the order of the k nearest.
__device__ __forceinline__ void exact_knn(FinalSmem &f, int metric, int dim, const float *rows, size_t ld,
                                          const int *ids, int self, const float *q, int n, int k)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = min(kSwBatch, (n + 3) / 4);   // few rows: all four warps
    const double margin = l2_margin(dim);
    for (int pass = 0; pass < 2; pass++) {
        if (tid == 0) f.risk = 0;
        __syncthreads();
        for (int b0 = warp * per; b0 < n; b0 += 4 * per) {
            const int nb = min(per, n - b0);
            const float *row[kSwBatch];
#pragma unroll
            for (int c = 0; c < kSwBatch; c++) row[c] = rows + (size_t)f.pos[b0 + min(c, nb - 1)] * ld;
            double d = pass == 0 ? exact_batch<false>(metric, dim, row, nb, q, f.ts[warp], lane)
                                 : exact_batch<true>(metric, dim, row, nb, q, f.ts[warp], lane);
            if (lane < nb) {
                const int p = f.pos[b0 + lane];
                if (p == self) d = 0.0;
                f.d[b0 + lane] = d;
                f.id[b0 + lane] = ids[p];
                if (pass == 0 && metric == kL2 && rounds_riskily(d, margin)) f.risk = 1;
            }
        }
        __syncthreads();
        sort_hits(f, n);
        if (metric != kL2 || pass == 1) break;
        for (int j = tid; j + 1 < n && j < k; j += 128) {
            const double a = f.d[j], b = f.d[j + 1];
            if (b != 0.0 && b - a <= (a + b) * margin) f.risk = 1;   // which comes first is open
        }
        __syncthreads();
        const int again = f.risk;
        __syncthreads();
        if (!again) break;
    }
}

// Ring bounds: the rows of the cut nodes that some query of each tile can
// reach, appended to the tiles' row lists (nrows zeroed by the caller).
void sweep_cut_launch(const SweepArgs &s, int ntiles, cudaStream_t st);

// The string sweep (edit distance); as run_sweep.
int run_sweep_edit(gts_index *idx, const SearchArgs &a, cudaStream_t st, int *done, const int4 **items, int *n_left);

}  // namespace gts
