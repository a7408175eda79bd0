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
    const int *cut, *anc, *anc_idx;
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
    int *ctr;                           // [0] item counter, [1] queries left over
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

// One step of the F32 sites' sum, r = (float)((double)r + pow(e, 2)), as one
// fused multiply-add: both round r + e^2 once, except that the reference's
// FP64 sum carries up to 2 ulp of the term and its own rounding, so the two
// may part where r + e^2 lies within 2^-50 of a float rounding midpoint.  The
// remainder e^2 + (r - f) is known to 2^-23 of itself when r >= f / 2 (the
// difference is then exact), which tells all but about 2^-19 of the steps
// apart; the few steps whose square is the larger part go through FP64.
__device__ __forceinline__ float add_square(float r, float e, bool &risk)
{
    const float f = fmaf(e, e, r);
    if (r < 0.5f * f) {
        const double t = (double)e * (double)e, s2 = (double)r + t;
        const float g = __double2float_rn(s2);
        const double gd = g, up = (double)__int_as_float(__float_as_int(g) + (s2 > gd ? 1 : -1));
        if (s2 != gd && fabs(s2 - 0.5 * (gd + up)) <= t * 8.9e-16 + s2 * 4.5e-16) risk = true;
        return g;
    }
    const float rem = fabsf(fmaf(e, e, r - f));
    const int bits = __float_as_int(f);
    const float half = __int_as_float((bits & 0x7f800000) - (24 << 23));   // half an ulp of f
    // below 2^-90 or past the floats the remainder is not reliable; at a power
    // of two the spacing below is half as wide
    if (fabsf(rem - half) <= half * 3e-6f || (e != 0.f && ((bits & 0x7fffff) == 0 || !(f > 1e-27f && f < 3e38f)))) risk = risk || e != 0.f;
    return f;
}

// The reference's value of up to kSwBatch rows against the query, row c's on
// lane c: the lanes make the terms of 32 dimensions of each row (coalesced),
// then lane c adds row c's in order.  F64 (kNN) or F32 (range) accumulation
// as dist_row_f64 / dist_row_f32.
//
// L2 terms: the reference's pow(e, 2) is within 2 ulp of the square, which is
// exact in FP64 for a float e and costs a multiplication (pow: 0.5 per clock
// and SM, which made it most of these kernels' time).  POW = false adds the
// squares.  F64: the caller checks that the sums are clear of everything they
// decide (l2_margin).  F32: see add_square; a step that may round differently
// sets *risky: that row wants POW = true.
template <bool F64, bool POW>
__device__ __forceinline__ double exact_batch(int metric, int dim, const float *const (&row)[kSwBatch], int n,
                                              const float *q, double (*ts)[33], int lane, bool *risky)
{
    double r = 0.0;
    float rf = 0.f;
    bool risk = false;
    float x[kSwBatch], y = lane < dim ? q[lane] : 0.f;
#pragma unroll
    for (int c = 0; c < kSwBatch; c++) x[c] = c < n && lane < dim ? __ldg(row[c] + lane) : 0.f;
    for (int c0 = 0; c0 < dim; c0 += 32) {
#pragma unroll
        for (int c = 0; c < kSwBatch; c++)
            if (c < n) {
                const float e = x[c] - y;
                if (!F64 && !POW) reinterpret_cast<float *>(ts[c])[lane] = metric == kL2 ? e : fabsf(e);
                else ts[c][lane] = metric != kL2 ? (double)fabsf(e) : (POW ? pow(e, 2) : (double)e * (double)e);
            }
        // the next 32 dimensions are on their way while lane c adds these
        const int j = c0 + 32 + lane;
        y = j < dim ? q[j] : 0.f;
#pragma unroll
        for (int c = 0; c < kSwBatch; c++) x[c] = c < n && j < dim ? __ldg(row[c] + j) : 0.f;
        __syncwarp();
        if (lane < n) {
            const int m = min(32, dim - c0);
            if (!F64 && !POW) {
                const float *e = reinterpret_cast<const float *>(ts[lane]);
                if (metric == kL2) {
#pragma unroll 4
                    for (int u = 0; u < m; u++) rf = add_square(rf, e[u], risk);
                } else if (metric == kL1) {
                    for (int u = 0; u < m; u++) rf += e[u];
                } else {
                    for (int u = 0; u < m; u++)
                        if (e[u] > rf) rf = e[u];
                }
                r = rf;
            } else {
                const double *e = ts[lane];
                if (metric == kLinf) {
                    for (int u = 0; u < m; u++)
                        if (e[u] > r) r = e[u];
                } else if (F64) {
#pragma unroll 8
                    for (int u = 0; u < m; u++) r += e[u];
                } else {
                    for (int u = 0; u < m; u++) rf += e[u];   // POW: L2
                }
            }
        }
        __syncwarp();
    }
    *risky = risk;
    if (metric == kLinf) return r;
    if (F64) return metric == kL2 ? pow(r, 0.5) : r;
    if (metric == kL2) rf = pow(rf, 0.5);
    return (double)rf;
}

// The reference's range value of up to kSwBatch rows, row c's on lane c.
__device__ __forceinline__ double range_batch(int metric, int dim, const float *const (&row)[kSwBatch], int n,
                                              const float *q, double (*ts)[33], int lane)
{
    bool risky;
    double d = exact_batch<false, false>(metric, dim, row, n, q, ts, lane, &risky);
    if (__any_sync(0xffffffffu, risky)) d = exact_batch<false, true>(metric, dim, row, n, q, ts, lane, &risky);
    return d;
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
            bool risky;
            double d = pass == 0 ? exact_batch<true, false>(metric, dim, row, nb, q, f.ts[warp], lane, &risky)
                                 : exact_batch<true, true>(metric, dim, row, nb, q, f.ts[warp], lane, &risky);
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
