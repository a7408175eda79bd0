// search_warp.cu -- range counts of few-dimensional rows, one query per warp.
//
// Up to kLaneRowDim dimensions the ring bounds leave a query some dozens of
// nodes and a few thousand objects of a few bytes each (40 nodes and 1,850
// objects per query on 10,000,000 points of the plane).  A CTA per query
// (search.cu) spends its time in barriers there: 14.3 ms for 100,000 queries,
// 0.02 of the HBM rate.  Here a warp walks the tree by itself:
//
//   * up to 32 internal nodes per step, one per lane.  A lane computes its
//     node's pivot distance and goes through the node's children (one 16-byte
//     record each); children that stay and have children themselves go to the
//     warp's stack, childless ones are neighbours in tree order and add up to
//     one run of rows per lane;
//   * the warp then goes over the runs, 32 rows at a time, with thresholds on
//     the unrooted value; the few rows between them get the reference's own
//     arithmetic at once.
//
// The stack cannot overflow: a step takes only as many nodes as their
// children have room for, and one node at a time needs no more room than the
// tree's height times its order.
#include <algorithm>
#include <cfloat>
#include "search.cuh"

namespace gts {

namespace {

constexpr int kWsWarps = 8;       // queries per CTA
constexpr int kWsStack = 512;     // pending internal nodes per query
constexpr int kWsReserve = 160;   // room for one path of the tree, order <= kWsOrder
constexpr int kWsOrder = 16;

template <int M>
__device__ __forceinline__ float ws_value(const float *row, const float (&q)[kLaneRowDim], int dim)
{
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < kLaneRowDim; j++) {
        if (j >= dim) break;
        const float d = __ldg(row + j) - q[j];
        if (M == kL2) v = fmaf(d, d, v);
        else if (M == kL1) v += fabsf(d);
        else v = fmaxf(v, fabsf(d));
    }
    return v;
}

template <int M>
__global__ void __launch_bounds__(32 * kWsWarps) k_search_warp(SearchArgs a, const int4 *__restrict__ nodes)
{
    __shared__ int stacks[kWsWarps][kWsStack];
    const DevTree &t = a.t;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    int *stack = stacks[warp];
    const int O = t.order, dim = t.dim;
    const bool timed = a.mode == kModeRangeTimed;
    const bool by_data = a.qrows != nullptr;
    const float r = a.r, rel = a.rel_eps * 1.25f, abs_eps = a.abs_eps * 1.25f;
    // v < vlow: certainly within r; v > vthr (or NaN): certainly not, for any
    // order of summation (value_bounds_f)
    const float g = 2.f * f32_sum_rel_bound(dim + 32) + 4.f * 5.9604645e-8f;
    float vlow, vthr;
    if (M == kL2) {
        vlow = r * r * (1.f - 4e-6f) / (1.f + g);
        vthr = r * r * (1.f + 4e-6f) / (1.f - g) + 4e-36f;
        if (vlow < 1e-30f) vlow = -1.f;
    } else {
        vlow = r * (1.f - 2e-6f) / (1.f + (M == kL1 ? g : 0.f));
        vthr = r * (1.f + 2e-6f) / (1.f - (M == kL1 ? g : 0.f));
    }
    unsigned long long n_obj = 0, n_piv = 0, n_exact = 0, n_done = 0;
    for (;;) {
        int w = 0;
        if (lane == 0) w = atomicAdd(a.counter, 1);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= a.qnum) break;
        const int4 item = a.items_in ? a.items_in[w] : make_int4(w, 0, 0, 0);
        const int q = item.x;
        if (q < 0) continue;   // an unused item slot
        const int qid = by_data ? -1 : a.qids[q];
        if (!by_data && (qid < 0 || qid >= t.num)) {
            if (lane == 0) {
                atomicMax(a.status, (int)kKsBadQuery);
                a.counts[q] = -1;
                if (timed) a.counts2[q] = -1;
            }
            continue;
        }
        const float *src = by_data ? a.qrows + (size_t)q * dim : t.rows + (size_t)qid * dim;
        float qv[kLaneRowDim];
#pragma unroll
        for (int j = 0; j < kLaneRowDim; j++) qv[j] = j < dim ? src[j] : 0.f;
        const int self = by_data ? -1 : t.pos_of_id[qid];
        const int tq = timed ? a.qtime[q] : 0;
        int cnt = 0, cnt2 = 0, top = 0, since = 0;   // since: rows gone over since the last hand-over
        auto hit = [&](int pos) {
            if (!timed) {
                cnt++;
                return;
            }
            const int id = t.id_list[pos];
            for (int e = a.ent_off[id], e1 = a.ent_off[id + 1]; e < e1; e++) {
                const int4 v = a.ents[e];
                cnt += (v.x < tq && tq < v.y) ? 1 : 0;
                cnt2 += (v.z < tq && tq < v.w) ? 1 : 0;
            }
        };
        auto rows = [&](int start, int len) {   // the warp over one run
            for (int o = lane; o < len; o += 32) {
                const int pos = start + o;
                if (pos == self) {   // the query object is at distance 0
                    hit(pos);
                    continue;
                }
                const float *row = t.trows + (size_t)pos * dim;
                const float v = ws_value<M>(row, qv, dim);
                if (v < vlow) {
                    hit(pos);
                } else if (v <= vthr) {
                    n_exact++;
                    if (dist_row_f32(row, src, dim, M) <= r) hit(pos);
                }
            }
        };
        const int4 root = nodes[item.y];   // (min_dis bits, size, first position, pivot)
        if (root.w < 0) {
            rows(root.z + item.z, root.y - item.z);
            if (lane == 0) n_obj += root.y - item.z;
        } else {
            if (lane == 0) stack[0] = item.y;
            top = 1;
        }
        __syncwarp();
        while (top > 0) {
            if (a.split_objs > 0 && since > a.split_objs && top > 32) {
                // hand all but the 32 newest nodes over as (query, node) items
                const int nd = top - 32;
                int base = 0;
                if (lane == 0) base = atomicAdd(a.n_items_out, nd);
                base = __shfl_sync(0xffffffffu, base, 0);
                if (base + nd <= a.items_cap) {
                    for (int i = lane; i < nd; i += 32) a.items_out[base + i] = make_int4(q, stack[i], 0, 0);
                    const int keep = stack[nd + lane];
                    __syncwarp();
                    stack[lane] = keep;
                    top = 32;
                    __syncwarp();
                } else {
                    // no room: keep them; mark this reservation's slots below the capacity unused
                    for (int i = base + lane; i < a.items_cap && i < base + nd; i += 32)
                        a.items_out[i] = make_int4(-1, 0, 0, 0);
                }
                since = 0;
            }
            const int n = min(min(32, top), max(1, (kWsStack - kWsReserve - top) / O));
            const bool have = lane < n;
            int node = 0;
            float dlo = 0.f, dhi = 0.f;
            if (have) {
                node = stack[top - 1 - lane];
                const int piv = nodes[node].w;
                if (piv != qid) {
                    const float v = ws_value<M>(t.rows + (size_t)piv * dim, qv, dim);
                    value_bounds_f(M, dim, M == kL2 ? v + 1e-36f : v, dlo, dhi);
                    if (M == kL2 && v < 1e-30f) dlo = 0.f;
                }
            }
            top -= n;
            __syncwarp();
            int start = 0, len = 0;   // the lane's run of rows
            const size_t c0 = (size_t)node * O + 1;
            int4 cur = have ? nodes[c0] : make_int4(0, 0, 0, -1);
            for (int i = 0; i < O; i++) {
                const int4 nxt = have && i + 1 < O ? nodes[c0 + i + 1] : make_int4(0, 0, 0, -1);
                bool stay = false;
                if (have && cur.y > 0) {
                    const float md = __int_as_float(cur.x);
                    float lb = fmaxf(md - dhi, 0.f);
                    if (i + 1 < O) lb = fmaxf(lb, dlo - __int_as_float(nxt.x));   // the next child starts where this one ends
                    stay = !(lb > r + abs_eps + rel * (dhi + fabsf(md) + r));
                }
                const bool inner = stay && cur.w >= 0;
                const unsigned m = __ballot_sync(0xffffffffu, inner);
                if (inner) stack[top + __popc(m & below)] = (int)(c0 + i);
                top += __popc(m);
                // childless children are neighbours in tree order; one that is
                // not the run's neighbour ends it
                const bool gap = stay && !inner && len > 0 && start + len != cur.z;
                for (unsigned todo = __ballot_sync(0xffffffffu, gap); todo; todo &= todo - 1) {
                    const int from = __ffs(todo) - 1;
                    const int l = __shfl_sync(0xffffffffu, len, from);
                    rows(__shfl_sync(0xffffffffu, start, from), l);
                    since += l;
                    if (lane == 0) n_obj += l;
                    if (lane == from) len = 0;
                }
                if (stay && !inner) {
                    if (len == 0) start = cur.z;
                    len += cur.y;
                }
                cur = nxt;
            }
            __syncwarp();
            for (unsigned todo = __ballot_sync(0xffffffffu, len > 0); todo; todo &= todo - 1) {
                const int from = __ffs(todo) - 1;
                const int l = __shfl_sync(0xffffffffu, len, from);
                rows(__shfl_sync(0xffffffffu, start, from), l);
                since += l;
                if (lane == 0) n_obj += l;
            }
            if (lane == 0) n_piv += n;
        }
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        cnt2 = __reduce_add_sync(0xffffffffu, cnt2);
        if (lane == 0) {
            const bool add = a.split_objs > 0 || a.items_in;
            if (add) atomicAdd(&a.counts[q], cnt);
            else a.counts[q] = cnt;
            if (timed) {
                if (add) atomicAdd(&a.counts2[q], cnt2);
                else a.counts2[q] = cnt2;
            }
            if (!a.items_in) n_done++;
        }
        __syncwarp();
    }
    if (a.stats) {
        n_exact = (unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)n_exact);
        if (lane == 0) {
            if (n_obj) atomicAdd(&a.stats[0], n_obj);
            if (n_piv) atomicAdd(&a.stats[1], n_piv);
            if (n_exact) atomicAdd(&a.stats[2], n_exact);
            if (n_done) atomicAdd(&a.stats[3], n_done);
        }
    }
}

template <int M>
int launch_warp(gts_index *idx, const SearchArgs &a, cudaStream_t st)
{
    int dev = 0, nsm = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    GTS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_search_warp<M>, 32 * kWsWarps, 0));
    const int grid = std::min(nsm * std::max(per_sm, 1), (a.qnum + kWsWarps - 1) / kWsWarps);
    k_search_warp<M><<<grid, 32 * kWsWarps, 0, st>>>(a, idx->node_rec);
    idx->kernel_launches++;
    GTS_CUDA_TRY(cudaGetLastError());
    return GTS_OK;
}

}  // namespace

// While most queries of a batch (or items of a hand-over) have a CTA of their
// own, 256 threads finish them sooner than a warp each: one query that reaches
// all of 4,000,000 points of the plane takes 0.84 ms there and 20.1 here, one
// of 0.1 % of 1,000,000 x 8 0.41 against 1.95.  Once they queue for the CTAs
// (296 resident on a B200) warps win: on small leaves from about half as many
// again (444 queries of 0.1 % over 1,000,000 x 8: 1.20 ms by CTAs, 1.26 by
// warps; 600: 1.40 and 1.30; of 10 %: 15.5 and 4.4), on leaves of more than a
// warp's rows, which keep a CTA's threads busy, from four times as many (888
// queries: 3.1 and 4.0, 1,200: 4.3 and 4.0).
constexpr int kWsLeafRows = 32;

bool warp_search_takes(const gts_index *idx, const SearchArgs &a)
{
    if (a.mode != kModeRangeCount && a.mode != kModeRangeTimed) return false;
    const bool wide_leaves = idx->num > (long long)kWsLeafRows * std::max(idx->nleaf, 1);
    if (2 * a.qnum < (wide_leaves ? 8 : 3) * idx->cta_resident[1]) return false;
    const bool metric = idx->metric == kL2 || idx->metric == kL1 || idx->metric == kLinf;
    // radii whose square leaves FP32's range, or negative ones, stay with the CTA traversal
    return metric && idx->dim <= kLaneRowDim && idx->params.tree_order <= kWsOrder && !a.deleted &&
           !idx->plain_pinned[kModeRangeCount] && a.r >= 0.f && a.r <= 1e15f;
}

int launch_search_warp(gts_index *idx, const SearchArgs &a, cudaStream_t st)
{
    switch (idx->metric) {
    case kL2: return launch_warp<kL2>(idx, a, st);
    case kL1: return launch_warp<kL1>(idx, a, st);
    default: return launch_warp<kLinf>(idx, a, st);
    }
}

}  // namespace gts
