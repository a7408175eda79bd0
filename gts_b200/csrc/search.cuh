// search.cuh -- what the plain form's two searches share: the per-query tree
// traversal (search.cu) and the batched sweep (sweep.cu).
#pragma once
#include "index.cuh"

namespace gts {

constexpr int kMaxK = 256;
constexpr int kLaneRowDim = 8;        // up to this dimension a lane filters a whole row

enum SearchMode { kModeKnn = 0, kModeRangeCount = 1, kModeRangeIds = 2, kModeRangeTimed = 3 };

struct SearchArgs {
    DevTree t;
    const int *qids;
    int qnum;
    int mode;
    int k;
    float r;
    float *kth;
    int *ids;
    float *dists;
    int *counts;
    const int *offsets;
    int *rids;
    float *rdists;
    const uint32_t *deleted;
    int *counter;
    int *status;
    // kNN seeded by the learned radius (nullable): squared radius per query
    // (float bits); a query with fewer than k objects inside is listed in
    // fail / n_fail instead of answered
    const int *seed_r2_bits;
    int *fail, *n_fail;
    unsigned long long *stats;   // [objects filtered, pivots evaluated, exact values, queries]
    // kModeRangeTimed: the query's operation index; per object id its
    // entries ents[ent_off[id] .. ent_off[id + 1]) as (tree_from, tree_to,
    // cache_from, cache_to), live in the tree at t when tree_from < t <
    // tree_to and in the cache list when cache_from < t < cache_to; counts
    // receives the tree part, counts2 the cache part
    const int *qtime;
    const int *ent_off;
    const int4 *ents;
    int *counts2;
    // queries given as data instead of ids (nullable): rows [qnum][dim], or
    // strings [qnum][109] with lengths; such a query is no object of the
    // index (no self match)
    const float *qrows;
    const char *qstrs;
    const int *qlens;
    // (query, node) work items, range counts only (count and timed modes):
    // items_in (nullable) are (query, node, first unverified object, lower
    // bound bits) handed over by an earlier launch; n_items_in of them are
    // the work units instead of the queries.  A query that has verified more
    // than split_objs objects in one CTA since its last hand-over gives all
    // but its kBatch newest stack entries to items_out (capacity items_cap,
    // count in *n_items_out; entries with query -1 are unused), so the next
    // launch spreads its subtrees over every CTA.  With splitting on, counts
    // are added atomically (the caller zeroes them first).
    const int4 *items_in;
    int4 *items_out;
    int *n_items_out;
    int items_cap;
    int split_objs;   // 0: no hand-over
    // count_objs > 0: answers nothing; query w * count_step walks the inner
    // nodes only and adds the objects of the leaves it reaches, at most
    // count_objs, to *reached
    int count_objs, count_step;
    unsigned long long *reached;
    float rel_eps;   // relative pruning slack
    float abs_eps;   // absolute pruning slack
};

// The pruning slacks and the handle's device pointers of a search.
void fill_search_args(gts_index *idx, SearchArgs &a);

// Range counts of up to kLaneRowDim dimensions, a query per warp
// (search_warp.cu).
bool warp_search_takes(const gts_index *idx, const SearchArgs &a);
int launch_search_warp(gts_index *idx, const SearchArgs &a, cudaStream_t st);

// Whether the batched sweep of rows is one for this batch, by its sizes alone.
bool sweep_takes(const gts_index *idx, const SearchArgs &a);

// The batched sweep (sweep.cu).  *done = 1: it answered every query of the
// batch except those it lists (query, 0, 0, 0) in items[0 .. *n_left), which
// the traversal answers; *done = 0: the batch is not one it takes.
int run_sweep(gts_index *idx, const SearchArgs &a, cudaStream_t st, int *done, const int4 **items, int *n_left);

// Warp-cooperative FP32 partial value of a row against the query:
// L2 -> sum of squares, L1 -> sum of |diff|, Linf -> max |diff| (exact).
__device__ __forceinline__ float warp_row_value(const float *__restrict__ row,
                                                const float *__restrict__ q, int dim, int metric,
                                                int lane)
{
    float acc = 0.f;
    if ((dim & 3) == 0) {
        const float4 *r4 = reinterpret_cast<const float4 *>(row);
        const float4 *q4 = reinterpret_cast<const float4 *>(q);
        for (int j = lane; j < (dim >> 2); j += 32) {
            float4 x = __ldg(r4 + j), y = q4[j];
            float d0 = x.x - y.x, d1 = x.y - y.y, d2 = x.z - y.z, d3 = x.w - y.w;
            if (metric == kL2) {
                acc = fmaf(d0, d0, acc); acc = fmaf(d1, d1, acc);
                acc = fmaf(d2, d2, acc); acc = fmaf(d3, d3, acc);
            } else if (metric == kL1) {
                acc += fabsf(d0) + fabsf(d1) + fabsf(d2) + fabsf(d3);
            } else {
                acc = fmaxf(acc, fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fmaxf(fabsf(d2), fabsf(d3))));
            }
        }
    } else {
        for (int j = lane; j < dim; j += 32) {
            float d0 = __ldg(row + j) - q[j];
            if (metric == kL2) acc = fmaf(d0, d0, acc);
            else if (metric == kL1) acc += fabsf(d0);
            else acc = fmaxf(acc, fabsf(d0));
        }
    }
    return metric == kLinf ? warp_max(acc) : warp_sum(acc);
}

// R rows at once (independent loads in flight): out[u] as warp_row_value.
template <int R>
__device__ __forceinline__ void warp_row_values(const float *const (&rows)[R], const float *__restrict__ q,
                                                int dim, int metric, int lane, float (&out)[R])
{
    float acc[R];
#pragma unroll
    for (int u = 0; u < R; u++) acc[u] = 0.f;
    if ((dim & 3) == 0) {
        const float4 *q4 = reinterpret_cast<const float4 *>(q);
        for (int j = lane; j < (dim >> 2); j += 32) {
            float4 x[R];
#pragma unroll
            for (int u = 0; u < R; u++) x[u] = __ldg(reinterpret_cast<const float4 *>(rows[u]) + j);
            const float4 y = q4[j];
#pragma unroll
            for (int u = 0; u < R; u++) {
                float d0 = x[u].x - y.x, d1 = x[u].y - y.y, d2 = x[u].z - y.z, d3 = x[u].w - y.w;
                if (metric == kL2) {
                    acc[u] = fmaf(d0, d0, acc[u]); acc[u] = fmaf(d1, d1, acc[u]);
                    acc[u] = fmaf(d2, d2, acc[u]); acc[u] = fmaf(d3, d3, acc[u]);
                } else if (metric == kL1) {
                    acc[u] += fabsf(d0) + fabsf(d1) + fabsf(d2) + fabsf(d3);
                } else {
                    acc[u] = fmaxf(acc[u], fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fmaxf(fabsf(d2), fabsf(d3))));
                }
            }
        }
    } else {
        for (int j = lane; j < dim; j += 32) {
            float x[R];
#pragma unroll
            for (int u = 0; u < R; u++) x[u] = __ldg(rows[u] + j);
            const float y = q[j];
#pragma unroll
            for (int u = 0; u < R; u++) {
                float d0 = x[u] - y;
                if (metric == kL2) acc[u] = fmaf(d0, d0, acc[u]);
                else if (metric == kL1) acc[u] += fabsf(d0);
                else acc[u] = fmaxf(acc[u], fabsf(d0));
            }
        }
    }
#pragma unroll
    for (int u = 0; u < R; u++) out[u] = metric == kLinf ? warp_max(acc[u]) : warp_sum(acc[u]);
}

// Interval [lo, hi] that contains both exact leaf values (F32 and F64
// sites) given the FP32 warp value v.
__device__ __forceinline__ void value_bounds(int metric, int dim, float v, double &lo, double &hi)
{
    if (metric == kLinf) {   // max of exactly rounded |diff|: exact
        lo = hi = (double)v;
        return;
    }
    double g = 2.0 * (double)f32_sum_rel_bound(dim + 32) + 4.0 * 5.9604645e-8;
    double vl = (double)v * (1.0 - g), vh = (double)v * (1.0 + g);
    if (metric == kL2) {
        lo = sqrt(vl > 0 ? vl : 0.0) * (1.0 - 1e-7);
        hi = sqrt(vh) * (1.0 + 1e-7);
    } else {
        lo = vl;
        hi = vh;
    }
}

// value_bounds in FP32: the products and square roots add at most a few
// ulps, covered by the extra 4e-7 / 2e-7 relative margins.
__device__ __forceinline__ void value_bounds_f(int metric, int dim, float v, float &lo, float &hi)
{
    if (metric == kLinf) {   // max of exactly rounded |diff|: exact
        lo = hi = v;
        return;
    }
    const float g = 2.f * f32_sum_rel_bound(dim + 32) + 4.f * 5.9604645e-8f;
    const float vl = v * (1.f - g), vh = v * (1.f + g);
    if (metric == kL2) {
        lo = sqrtf(fmaxf(vl, 0.f)) * (1.f - 4e-7f);
        hi = sqrtf(vh) * (1.f + 4e-7f);
    } else {
        lo = vl * (1.f - 2e-7f);
        hi = vh * (1.f + 2e-7f);
    }
}

}  // namespace gts
