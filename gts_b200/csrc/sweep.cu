// sweep.cu -- the plain form's batched search: tiles of queries against tiles
// of rows.
//
// The traversal (search.cu) reads every leaf object once per query that
// reaches it.  On data of more than a few dimensions the ring bounds leave a
// large part of the objects to every query (467,000 of 1,000,000 x 128 at
// k = 8), so a batch reads the same rows over and over: 239 GB for 1,000
// queries.  Here 128 queries share each row they read:
//
//   * seeds (kNN): a query's k-th distance is bounded by the k-th smallest
//     upper bound over the objects around its place in the tree order;
//   * the ring bounds of the tree (nodeProcessKnn / nodeProcessRnn,
//     search_v2.cuh:131-141, 181-192) are applied to the topmost nodes of at
//     most kCutSize objects ("cut" nodes): a tile of queries keeps a cut node
//     that some query of the tile can reach, and the rows of its cut nodes
//     become tiles of 128;
//   * the filter multiplies out FP32 distances of 128 queries x 128 rows,
//     16 dimensions at a time, from registers.  A partial sum of non-negative
//     terms is a lower bound, so after each stage the pairs still within
//     their query's bound are counted: few of them leave the tile and are
//     finished one by one, none ends it.  On clustered data one stage of
//     128 dimensions settles nearly every tile;
//   * pairs within the bound are listed per query; their bounds, then the
//     reference's own arithmetic (metric.cuh), decide, as in the traversal.
//
// Every bound is the traversal's (search.cuh), for any order of summation, so
// the answers are the traversal's.  A query whose list does not hold its
// candidates goes to the traversal.  The angle metric has no partial bound;
// its three sums run in the reference's order, so the filter has the exact
// value.
#include <cub/device/device_radix_sort.cuh>
#include <algorithm>
#include <cfloat>
#include <climits>
#include "sweep.cuh"

namespace gts {

namespace {

constexpr int kSwThreads = 256;
constexpr int kSwRows = 128;           // rows per tile
constexpr int kSwK = 16;               // dimensions per stage
constexpr int kSwLd = kSwK + 4;        // row stride in shared memory (16-byte reads of 8 rows miss each other's banks)
constexpr int kSwList = 2048;          // pairs a tile may finish one by one
constexpr int kSwWindow = 1024;        // objects around a query's place that bound its k-th distance
constexpr int kSwMaxTiles = 32;        // query tiles per run
constexpr int kSwFew = 32;             // up to so many queries take the small tile
constexpr int kSwSample = 16;          // the sample pass looks at every 16th row
constexpr int kSwSampleMin = 1 << 16;  // objects from which on it pays
constexpr int kSwRounds = 3;           // further passes over kNN queries whose lists overflowed
constexpr int kSwHitCap = 16384;       // hits per query of a range-ids call at most

__device__ __forceinline__ void sw_cp16(void *dst, const void *src, int bytes)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sw_cp4(void *dst, const void *src, int bytes)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// Sum over the CTA of a value per warp lane set (all threads get it).
__device__ __forceinline__ float cta_row_sum(float v, float *red, int metric)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = metric == kLinf ? warp_max(v) : warp_sum(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float r = 0.f;
    for (int w = 0; w < kSwThreads / 32; w++) r = metric == kLinf ? fmaxf(r, red[w]) : r + red[w];
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------- seeds

__device__ __forceinline__ const float *sw_query_row(const SweepArgs &s, int q)
{
    return s.a.qrows ? s.a.qrows + (size_t)(s.q0 + q) * s.a.t.dim : s.a.t.rows + (size_t)s.a.qids[s.q0 + q] * s.a.t.dim;
}

// One CTA per query of the run: its place in the tree order (a query given as
// data goes down the rings its pivot distances fall into), and for kNN the
// k-th smallest upper bound over the kSwWindow objects around it.
__global__ void __launch_bounds__(kSwThreads) k_sw_seed(SweepArgs s, int window)
{
    extern __shared__ __align__(16) float sq[];   // the query row
    __shared__ uint32_t hib[kSwWindow];
    __shared__ int hist[256];
    __shared__ float red[kSwThreads / 32];
    __shared__ int s_node;
    const DevTree &t = s.a.t;
    const int q = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool by_data = s.a.qrows != nullptr;
    const int qid = by_data ? -1 : s.a.qids[s.q0 + q];
    if (!by_data && (qid < 0 || qid >= t.num)) {
        if (tid == 0) {
            atomicMax(s.a.status, (int)kKsBadQuery);
            s.key[q] = 0;
            s.seed[q] = 0.f;
        }
        return;
    }
    if (s.a.mode != kModeKnn && !by_data) {
        if (tid == 0) s.key[q] = t.pos_of_id[qid];
        return;
    }
    const float *src = sw_query_row(s, q);
    for (int j = tid; j < t.dim; j += kSwThreads) sq[j] = src[j];
    __syncthreads();
    float qn = 0.f;
    if (t.metric == kAngle) {
        float v = 0.f;
        for (int j = tid; j < t.dim; j += kSwThreads) v = fmaf(sq[j], sq[j], v);
        qn = sqrtf(cta_row_sum(v, red, kL2));
    }
    const float aeps = 4.f * (float)(t.dim + 32) * 5.9604645e-8f;   // cosines by any order of summation
    int pos = 0;
    if (!by_data) {
        pos = t.pos_of_id[qid];
    } else {
        int node = 0;
        while (t.node_pivot[node] >= 0) {
            const float *p = t.rows + (size_t)t.node_pivot[node] * t.dim;
            float v = 0.f, pn = 0.f;
            for (int j = tid; j < t.dim; j += kSwThreads) {
                const float x = p[j], d = x - sq[j];
                if (t.metric == kL2) v = fmaf(d, d, v);
                else if (t.metric == kL1) v += fabsf(d);
                else if (t.metric == kLinf) v = fmaxf(v, fabsf(d));
                else {
                    v = fmaf(x, sq[j], v);
                    pn = fmaf(x, x, pn);
                }
            }
            v = cta_row_sum(v, red, t.metric);
            if (t.metric == kL2) v = sqrtf(v);
            if (t.metric == kAngle) {
                pn = sqrtf(cta_row_sum(pn, red, kL2));
                v = acosf(fminf(fmaxf(v / (pn * qn), -1.f), 1.f)) * 57.2957795f;
            }
            if (tid == 0) {   // the last child that starts at or below the distance
                int at = -1;
                for (int i = 0; i < t.order; i++) {
                    const long c = (long)node * t.order + i + 1;
                    if (c >= t.max_node_num || !(t.node_flags[c] & kExists) || t.node_size[c] == 0) continue;
                    if (at < 0 || t.node_min_dis[c] <= v) at = (int)c;
                }
                s_node = at;
            }
            __syncthreads();
            const int next = s_node;
            __syncthreads();
            if (next < 0) break;
            node = next;
        }
        pos = t.node_lid[node] + t.node_size[node] / 2;
        if (pos >= t.num) pos = t.num - 1;
    }
    if (tid == 0) s.key[q] = pos;
    if (s.a.mode != kModeKnn) return;
    const int w = min(window, t.num), w0 = max(0, min(pos - w / 2, t.num - w));
    const int k = s.a.k;
    constexpr int kR = 8;
    for (int o = warp * kR; o < w; o += (kSwThreads / 32) * kR) {
        const float *rp[kR];
#pragma unroll
        for (int u = 0; u < kR; u++) rp[u] = t.trows + (size_t)(w0 + min(o + u, w - 1)) * t.dim;
        float v[kR];
        if (t.metric == kAngle) {
#pragma unroll
            for (int u = 0; u < kR; u++) v[u] = 0.f;
            for (int j = lane; j < t.dim; j += 32) {
                const float y = sq[j];
#pragma unroll
                for (int u = 0; u < kR; u++) v[u] = fmaf(__ldg(rp[u] + j), y, v[u]);
            }
#pragma unroll
            for (int u = 0; u < kR; u++) v[u] = warp_sum(v[u]);
        } else {
            warp_row_values<kR>(rp, sq, t.dim, t.metric, lane, v);
        }
        float mine = 0.f;
#pragma unroll
        for (int u = 0; u < kR; u++)
            if (lane == u) mine = v[u];
        if (lane < kR && o + lane < w) {
            const int p = w0 + o + lane;
            float hi;
            if (t.metric == kAngle) {
                const float c = mine / (s.tnorm[p] * qn) - aeps;
                hi = acosf(fminf(fmaxf(c, -1.f), 1.f)) * 57.2957795f * 1.00001f + 1e-3f;
                if (!(c == c)) hi = FLT_MAX;
            } else {
                hi = sw_hi(t.metric, t.dim, mine);
            }
            if (!by_data && t.id_list[p] == qid) hi = 0.f;
            hib[o + lane] = hi < FLT_MAX ? __float_as_uint(hi) : __float_as_uint(FLT_MAX);
        }
    }
    __syncthreads();
    float R = FLT_MAX;
    if (k <= w) R = __uint_as_float(cta_kth(hib, w, k, hist));
    if (tid == 0) {
        s.seed[q] = R;
        if (s.a.stats) atomicAdd(&s.a.stats[0], (unsigned long long)w);
    }
}

// The order to be sorted.
__global__ void k_sw_iota(int n, int *v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}

// Thresholds on the filter value for radius R: above vthr (angle: below) no
// bound admits the object, below vlow a range hit is certain.
__device__ __forceinline__ void sw_thresholds(const DevTree &t, float R, bool ok, float &vthr, float &vlow)
{
    vlow = -1.f;
    if (t.metric == kAngle) {
        vthr = 3.f;   // nothing passes
        if (ok) {
            const double deg = (double)R * (1.0 + 1e-5) + 1e-3;
            vthr = deg >= 180.0 ? -2.f : (float)(cos(deg * (3.14159265358979 / 180.0)) - 1e-6);
        }
        return;
    }
    vthr = -1.f;
    if (!ok) return;
    const double g = 2.0 * (double)f32_sum_rel_bound(t.dim + 32) + 4.0 * 5.9604645e-8;
    double hi, lo;
    if (t.metric == kL2) {
        hi = (double)R * R * (1.0 + 4e-6) / (1.0 - g) + 4.0 * kSwTiny;
        lo = (double)R * R * (1.0 - 4e-6) / (1.0 + g);
        if (lo < 1e-30) lo = -1.0;
    } else if (t.metric == kL1) {
        hi = (double)R * (1.0 + 2e-6) / (1.0 - g);
        lo = (double)R * (1.0 - 2e-6) / (1.0 + g);
    } else {
        hi = (double)R * (1.0 + 2e-6);
        lo = (double)R * (1.0 - 2e-6);
    }
    vthr = hi < FLT_MAX ? __double2float_ru(hi) : FLT_MAX;
    vlow = __double2float_rd(lo);
}

// One warp per sorted query slot: its row (zero padded), radius, thresholds
// on the filter value, and an empty candidate list (the query object itself
// first: its distance is 0 by definition, search_v2.cuh:338-340).  The pass's
// counters are cleared here too.
__global__ void __launch_bounds__(256) k_sw_query(SweepArgs s)
{
    const DevTree &t = s.a.t;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (blockIdx.x == 0) {
        for (int j = threadIdx.x; j < s.ntiles; j += 256) s.nrows[j] = 0;
        if (threadIdx.x == 0) s.ctr[0] = 0;
    }
    if (i >= s.Qp) return;
    const bool have = i < s.nq;
    const int q = !have ? -1 : (s.again ? s.again[s.q0 + i].x : s.q0 + (s.nq > 128 ? s.order[i] : i));   // in the batch
    if (lane == 0) s.bq[i] = q;
    const int qid = have && !s.a.qrows ? s.a.qids[q] : -1;
    const bool ok = have && (s.a.qrows || (qid >= 0 && qid < t.num));
    const float *src = !ok ? nullptr : (s.a.qrows ? s.a.qrows + (size_t)q * t.dim : t.rows + (size_t)qid * t.dim);
    for (int j = lane; j < s.ld; j += 32) s.qrow[(size_t)i * s.ld + j] = ok && j < t.dim ? src[j] : 0.f;
    if (lane == 0) {
        float R = -1.f;
        if (ok) R = s.a.mode != kModeKnn ? s.a.r : (s.again ? s.again_R[s.q0 + i] : s.seed[q - s.q0]);
        float vthr, vlow, qn = 0.f;
        if (have && !ok) atomicMax(s.a.status, (int)kKsBadQuery);
        if (ok && t.metric == kAngle) {
            float sa = 0.f;
            for (int j = 0; j < t.dim; j++) sa = fmaf(src[j], src[j], sa);
            sa = pow(sa, 0.5);
            qn = sa;
        }
        sw_thresholds(t, R, ok, vthr, vlow);
        s.R[i] = R;
        s.vthr[i] = vthr;
        s.vlow[i] = vlow;
        s.qnorm[i] = qn;
        const int self = ok && qid >= 0 ? t.pos_of_id[qid] : -1;
        s.self[i] = self;
        int n = 0;
        s.cnt[i] = 0;
        s.cnt2[i] = 0;
        if (self >= 0) {
            if (s.a.mode == kModeKnn || s.a.mode == kModeRangeIds) {
                s.cpos[(size_t)i * s.cap] = self;
                s.cv[(size_t)i * s.cap] = t.metric == kAngle ? 1.f : 0.f;
                n = 1;
            } else if (s.a.mode == kModeRangeCount) {
                s.cnt[i] = 1;
            } else {
                const int tq = s.a.qtime[q];
                int wt = 0, wc = 0;
                for (int e = s.a.ent_off[qid], e1 = s.a.ent_off[qid + 1]; e < e1; e++) {
                    const int4 v = s.a.ents[e];
                    wt += (v.x < tq && tq < v.y) ? 1 : 0;
                    wc += (v.z < tq && tq < v.w) ? 1 : 0;
                }
                s.cnt[i] = wt;
                s.cnt2[i] = wc;
            }
        }
        s.ccnt[i] = n;
    }
}

// ---------------------------------------------------------------- ring bounds

// The cut nodes that some query of tile blockIdx.y can reach: one thread per
// cut node (or piece of one: a warp went over a childless node of 20,000 strings
// by itself for 1.8 ms) keeps a mask of the tile's (at most 128) queries and walks its ancestors, as
// the traversal does from above.  The rows of the kept nodes of a CTA's 256
// are appended to the tile's row list.
__global__ void __launch_bounds__(256) k_sw_cut(SweepArgs s)
{
    __shared__ float sR[128];
    __shared__ int wsum[8], s_base;
    __shared__ uint32_t lok[4];
    const DevTree &t = s.a.t;
    const int tile = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q0 = tile * s.tq, nq = min(s.tq, s.nq - q0);
    if (tid < 128) sR[tid] = tid < nq ? s.R[q0 + tid] : 0.f;
    if (s.lens_ok && tid < 4) lok[tid] = reinterpret_cast<const uint32_t *>(s.lens_ok + tile)[tid];
    __syncthreads();
    const int i = blockIdx.x * 256 + tid;
    int size = 0, lid = 0;
    if (i < s.ncut) {
        const int2 piece = s.cut[i];
        const int node = piece.x;
        size = min(t.node_size[node] - piece.y, kCutSize);
        lid = t.node_lid[node] + piece.y;
        uint32_t m[4];
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const int n = nq - 32 * w;
            m[w] = n >= 32 ? 0xffffffffu : (n > 0 ? (1u << n) - 1u : 0u);
        }
        const float rel = s.a.rel_eps * 1.25f, abs_eps = s.a.abs_eps * 1.25f;
        for (int c = node; c > 0 && (m[0] | m[1] | m[2] | m[3]);) {
            const int p = (c - 1) / t.order;
            const float md = t.node_min_dis[c];
            const bool inner = c % t.order != 0;
            const float md2 = inner ? t.node_min_dis[c + 1] : 0.f;
            const size_t at = (size_t)s.anc_idx[p] * s.Qp + q0;
            const float4 *lo4 = reinterpret_cast<const float4 *>(s.dlo + at);
            const float4 *hi4 = reinterpret_cast<const float4 *>(s.dhi + at);
#pragma unroll
            for (int w = 0; w < 4; w++) {
                if (!m[w]) continue;
#pragma unroll 2
                for (int b = 0; b < 8; b++) {
                    if (!((m[w] >> (4 * b)) & 15u)) continue;
                    const float4 l = lo4[w * 8 + b], h = hi4[w * 8 + b];
                    const float lv[4] = {l.x, l.y, l.z, l.w}, hv[4] = {h.x, h.y, h.z, h.w};
                    uint32_t dead = 0;
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const float R = sR[w * 32 + b * 4 + u];
                        float lb = fmaxf(md - hv[u], 0.f);
                        if (inner) lb = fmaxf(lb, lv[u] - md2);
                        const float slack = abs_eps + rel * (hv[u] + fabsf(md) + (R < 1e30f ? R : 0.f));
                        if (lb > R + slack) dead |= 1u << u;
                    }
                    m[w] &= ~(dead << (4 * b));
                }
            }
            c = p;
        }
        if (!(m[0] | m[1] | m[2] | m[3])) size = 0;
    }
    if (s.sample > 1) {   // every sample-th position only
        const int first = (lid + s.sample - 1) / s.sample * s.sample;
        size = first < lid + size ? (lid + size - 1 - first) / s.sample + 1 : 0;
        lid = first;
    }
    // the warp goes over its kept nodes together; strings of lengths that no
    // query of the tile can match are left out (strings are not sampled)
    auto fits = [&](int pos) {
        const int n = min(max(t.tlens[pos], 0), 127);
        return (lok[n >> 5] >> (n & 31)) & 1u;
    };
    const unsigned mine = __ballot_sync(0xffffffffu, size > 0);
    int kept = size;
    unsigned kb[4] = {0, 0, 0, 0};   // the lane's node: which of its strings stay
    if (s.lens_ok)
        for (unsigned todo = mine; todo; todo &= todo - 1) {
            const int from = __ffs(todo) - 1;
            const int n = __shfl_sync(0xffffffffu, size, from), l = __shfl_sync(0xffffffffu, lid, from);
            unsigned b[4];
#pragma unroll
            for (int u = 0; u < 4; u++) b[u] = __ballot_sync(0xffffffffu, u * 32 + lane < n && fits(l + u * 32 + lane));
            if (lane == from) {
                kept = 0;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    kb[u] = b[u];
                    kept += __popc(b[u]);
                }
            }
        }
    int incl = kept;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int w = 0; w < 8; w++) {
            const int c = wsum[w];
            wsum[w] = run;
            run += c;
        }
        s_base = run ? atomicAdd(&s.nrows[tile], run) : 0;
    }
    __syncthreads();
    const int off = s_base + wsum[warp] + incl - kept;
    int *dst = s.rowpos + (size_t)tile * t.num;
    for (unsigned todo = mine; todo; todo &= todo - 1) {
        const int from = __ffs(todo) - 1;
        const int n = __shfl_sync(0xffffffffu, size, from), l = __shfl_sync(0xffffffffu, lid, from);
        int o = __shfl_sync(0xffffffffu, off, from);
        if (!s.lens_ok) {
            for (int j = lane; j < n; j += 32) dst[o + j] = l + j * s.sample;
            continue;
        }
        const unsigned below = (1u << lane) - 1u;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const unsigned b = __shfl_sync(0xffffffffu, kb[u], from);
            if ((b >> lane) & 1u) dst[o + __popc(b & below)] = l + u * 32 + lane;
            o += __popc(b);
        }
    }
}

// ---------------------------------------------------------------- tiles

template <int QI>
struct SweepSmem {
    float a[2][16 * QI * kSwLd], b[2][kSwRows * kSwLd];
    const float *rp[kSwRows];
    int pos[kSwRows];
    float vthr[16 * QI], vlow[16 * QI];
    int self[16 * QI];
    int cnt[16 * QI], cnt2[16 * QI];
    unsigned short list[kSwList];
    int item[2], nlist[2];
};

// 16 QI query rows from qrow and 128 rows at rp, dimensions k0 .. k0 + 15,
// zeros past the rows' dimensions.
template <int QI>
__device__ __forceinline__ void sw_stage(SweepSmem<QI> &s, int st, const float *qrow, int ld, int dim, int k0)
{
    for (int i = threadIdx.x; i < 16 * QI * 4; i += kSwThreads) {
        const int r = i >> 2, j = (i & 3) * 4;
        sw_cp16(s.a[st] + r * kSwLd + j, qrow + (size_t)r * ld + k0 + j, 16);
    }
    if ((dim & 3) == 0) {
        for (int i = threadIdx.x; i < kSwRows * 4; i += kSwThreads) {
            const int r = i >> 2, j = (i & 3) * 4, k = k0 + j;
            sw_cp16(s.b[st] + r * kSwLd + j, s.rp[r] + (k < dim ? k : 0), k < dim ? 16 : 0);
        }
    } else {
        for (int i = threadIdx.x; i < kSwRows * 16; i += kSwThreads) {
            const int r = i >> 4, j = i & 15, k = k0 + j;
            sw_cp4(s.b[st] + r * kSwLd + j, s.rp[r] + (k < dim ? k : 0), k < dim ? 4 : 0);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int M>
__device__ __forceinline__ float sw_term(float acc, float o, float q)
{
    if (M == kAngle) return fmaf(o, q, acc);
    const float d = o - q;
    return M == kL2 ? fmaf(d, d, acc) : (M == kL1 ? acc + fabsf(d) : fmaxf(acc, fabsf(d)));
}

template <int M, int QI>
__device__ __forceinline__ void sw_add(const float *a, const float *b, int tq, int to, float (&acc)[QI][8])
{
#pragma unroll
    for (int k = 0; k < kSwK; k += 4) {
        float4 o[8];
#pragma unroll
        for (int c = 0; c < 8; c++) o[c] = *reinterpret_cast<const float4 *>(b + (to + 16 * c) * kSwLd + k);
#pragma unroll
        for (int i = 0; i < QI; i++) {
            const float4 q = *reinterpret_cast<const float4 *>(a + (tq + 16 * i) * kSwLd + k);
#pragma unroll
            for (int c = 0; c < 8; c++) {
                acc[i][c] = sw_term<M>(acc[i][c], o[c].x, q.x);
                acc[i][c] = sw_term<M>(acc[i][c], o[c].y, q.y);
                acc[i][c] = sw_term<M>(acc[i][c], o[c].z, q.z);
                acc[i][c] = sw_term<M>(acc[i][c], o[c].w, q.w);
            }
        }
    }
}

// Pivot distance bounds of tile blockIdx.y's queries to 128 ancestors of the
// cut nodes: [nanc][Qp], queries fastest.
template <int M, int QI>
__global__ void __launch_bounds__(kSwThreads) k_sw_pivots(SweepArgs s)
{
    extern __shared__ __align__(16) unsigned char sw_smem[];
    SweepSmem<QI> &sm = *reinterpret_cast<SweepSmem<QI> *>(sw_smem);
    const DevTree &t = s.a.t;
    const int tid = threadIdx.x, tq = tid & 15, to = tid >> 4;
    const int a0 = blockIdx.x * kSwRows, q0 = blockIdx.y * 16 * QI;
    if (tid < kSwRows) {
        const int piv = t.node_pivot[s.anc[min(a0 + tid, s.nanc - 1)]];
        sm.pos[tid] = t.pos_of_id[piv];
        sm.rp[tid] = t.rows + (size_t)piv * t.dim;
    }
    __syncthreads();
    float acc[QI][8];
#pragma unroll
    for (int i = 0; i < QI; i++)
#pragma unroll
        for (int c = 0; c < 8; c++) acc[i][c] = 0.f;
    const int nc = s.ld / kSwK;
    const float *qrow = s.qrow + (size_t)q0 * s.ld;
    sw_stage<QI>(sm, 0, qrow, s.ld, t.dim, 0);
    for (int ch = 0; ch < nc; ch++) {
        if (ch + 1 < nc) {
            sw_stage<QI>(sm, (ch + 1) & 1, qrow, s.ld, t.dim, (ch + 1) * kSwK);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        sw_add<M, QI>(sm.a[ch & 1], sm.b[ch & 1], tq, to, acc);
        __syncthreads();
    }
    // the bounds, half of the pivots at a time through shared memory: written
    // out per accumulator they made the single CTA of a small batch take 35 us
    // at 64 dimensions, in a loop 17
    constexpr int kQ = 16 * QI, kLd = kQ + 1;
    float *v = &sm.a[0][0];
    static_assert(sizeof(sm.a) + sizeof(sm.b) >= sizeof(float) * 64 * kLd, "half a tile of values");
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
        for (int i = 0; i < QI; i++)
#pragma unroll
            for (int c = 0; c < 4; c++) v[(to + 16 * c) * kLd + tq + 16 * i] = acc[i][4 * h + c];
        __syncthreads();
        const int q = q0 + tid % kQ, self = s.self[q];
        const float qn = s.qnorm[q];
#pragma unroll 1
        for (int r = tid / kQ; r < 64; r += kSwThreads / kQ) {
            const int p = 64 * h + r;
            if (a0 + p >= s.nanc) break;
            const float x = v[r * kLd + tid % kQ];
            float lo, hi;
            if (M == kAngle) {
                lo = hi = (float)angle_of_cos_f64(x / (s.tnorm[sm.pos[p]] * qn));
            } else {
                lo = sw_lo(M, t.dim, x);
                hi = sw_hi(M, t.dim, x);
            }
            if (sm.pos[p] == self) lo = hi = 0.f;
            s.dlo[(size_t)(a0 + p) * s.Qp + q] = lo;
            s.dhi[(size_t)(a0 + p) * s.Qp + q] = hi;
        }
        __syncthreads();
    }
}

// A pair within its query's bound: kNN and range ids list it; range counts
// take it when it is certain and list it for the exact value otherwise.
template <int M, int QI>
__device__ __forceinline__ void sw_emit(const SweepArgs &s, SweepSmem<QI> &sm, int q0, int q, int r, float v)
{
    const int pos = sm.pos[r];
    if (pos == sm.self[q]) return;
    const int mode = s.a.mode;
    if (mode == kModeRangeCount || mode == kModeRangeTimed) {
        bool in = v < sm.vlow[q];
        if (M == kAngle) {
            if (!(angle_of_cos_f32(v) <= s.a.r)) return;
            in = true;
        }
        if (in) {
            if (mode == kModeRangeCount) {
                atomicAdd(&sm.cnt[q], 1);
            } else {
                const int id = s.a.t.id_list[pos], tq = s.a.qtime[s.bq[q0 + q]];
                int wt = 0, wc = 0;
                for (int e = s.a.ent_off[id], e1 = s.a.ent_off[id + 1]; e < e1; e++) {
                    const int4 x = s.a.ents[e];
                    wt += (x.x < tq && tq < x.y) ? 1 : 0;
                    wc += (x.z < tq && tq < x.w) ? 1 : 0;
                }
                if (wt) atomicAdd(&sm.cnt[q], wt);
                if (wc) atomicAdd(&sm.cnt2[q], wc);
            }
            return;
        }
    }
    const int at = atomicAdd(&s.ccnt[q0 + q], 1);
    if (at < s.cap) {
        s.cpos[(size_t)(q0 + q) * s.cap + at] = pos;
        s.cv[(size_t)(q0 + q) * s.cap + at] = v;
    }
}

// The filter: persistent CTAs take (row tile, query tile) items, row tiles
// outermost so that the query tiles meet the same rows in L2.
template <int M, int QI>
__global__ void __launch_bounds__(kSwThreads, QI == 8 ? 2 : 3) k_sw_tile(SweepArgs s)
{
    extern __shared__ __align__(16) unsigned char sw_smem[];
    SweepSmem<QI> &sm = *reinterpret_cast<SweepSmem<QI> *>(sw_smem);
    const DevTree &t = s.a.t;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tq = tid & 15, to = tid >> 4;
    const int nc = s.ld / kSwK;
    const bool counts = s.a.mode == kModeRangeCount || s.a.mode == kModeRangeTimed;
    int maxj = 0;
    for (int i = 0; i < s.ntiles; i++) maxj = max(maxj, (s.nrows[i * (16 * QI) / 128] + kSwRows - 1) / kSwRows);
    // a pair finished alone costs a warp about 30 + dim / 4 instructions, a
    // stage of the tile QI * 8 * 16 * 2 of each of its eight warps
    const int alone = 30 + t.dim / 4, stage_cost = QI * 8 * kSwK * 2 * (kSwThreads / 32);
    if (tid == 0) sm.item[0] = atomicAdd(&s.ctr[0], 1);
    if (tid < 16 * QI) sm.cnt[tid] = sm.cnt2[tid] = 0;
    unsigned long long pairs = 0;
    for (int it = 0;; it++) {
        __syncthreads();
        const int id = sm.item[it & 1], j = id / s.ntiles, tile = id - j * s.ntiles;
        if (j >= maxj) break;
        if (tid == 0) sm.item[(it + 1) & 1] = atomicAdd(&s.ctr[0], 1);
        const int rt = tile * (16 * QI) / 128;   // the row list is kept per 128 queries
        const int nr = min(kSwRows, s.nrows[rt] - j * kSwRows);
        if (nr <= 0) continue;
        const int q0 = tile * 16 * QI;
        if (tid < kSwRows) {
            const int p = s.rowpos[(size_t)rt * t.num + (size_t)j * kSwRows + min(tid, nr - 1)];
            sm.pos[tid] = p;
            sm.rp[tid] = t.trows + (size_t)p * t.dim;
        }
        if (tid < 16 * QI) {
            sm.vthr[tid] = s.vthr[q0 + tid];
            sm.vlow[tid] = s.vlow[q0 + tid];
            sm.self[tid] = s.self[q0 + tid];
        }
        if (tid == 0) {
            sm.nlist[0] = sm.nlist[1] = 0;
            pairs += (unsigned long long)nr * max(0, min(16 * QI, s.nq - q0));
        }
        __syncthreads();
        const float *qrow = s.qrow + (size_t)q0 * s.ld;
        float acc[QI][8];
#pragma unroll
        for (int i = 0; i < QI; i++)
#pragma unroll
            for (int c = 0; c < 8; c++) acc[i][c] = 0.f;
        sw_stage<QI>(sm, 0, qrow, s.ld, t.dim, 0);
        bool whole = true;   // the tile ran through all dimensions
        int n = 0;           // else: pairs listed to be finished one by one
        for (int ch = 0; ch < nc; ch++) {
            // only the angle metric is sure to need the next stage
            if (M == kAngle && ch + 1 < nc) {
                sw_stage<QI>(sm, (ch + 1) & 1, qrow, s.ld, t.dim, (ch + 1) * kSwK);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            if (M != kAngle && ch > 0 && ch + 1 < nc)
                sw_stage<QI>(sm, (ch + 1) & 1, qrow, s.ld, t.dim, (ch + 1) * kSwK);
            sw_add<M, QI>(sm.a[ch & 1], sm.b[ch & 1], tq, to, acc);
            if (M == kAngle || ch + 1 == nc) {
                __syncthreads();
                continue;
            }
            // list the pairs still within their bounds; too many of them to
            // finish one by one: drop the list and take the next stage
            const int most = (int)min((long)kSwList, (long)(nc - 1 - ch) * stage_cost / alone);
            int *nlist = &sm.nlist[ch & 1];
#pragma unroll
            for (int i = 0; i < QI; i++) {
                const float th = sm.vthr[tq + 16 * i];
                float mn = acc[i][0];
#pragma unroll
                for (int c = 1; c < 8; c++) mn = fminf(mn, acc[i][c]);
                if (mn <= th && *(volatile int *)nlist <= most) {
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        if (acc[i][c] <= th && to + 16 * c < nr) {
                            const int at = atomicAdd(nlist, 1);
                            if (at < kSwList) sm.list[at] = (unsigned short)((tq + 16 * i) << 7 | (to + 16 * c));
                        }
                }
            }
            __syncthreads();
            n = *nlist;
            if (tid == 0) sm.nlist[(ch + 1) & 1] = 0;
            if (n <= most) {
                whole = false;
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                break;
            }
            if (ch == 0 && nc > 1) sw_stage<QI>(sm, 1, qrow, s.ld, t.dim, kSwK);
        }
        if (whole) {
#pragma unroll
            for (int i = 0; i < QI; i++) {
                const int q = tq + 16 * i;
                const float th = sm.vthr[q];
                const float qn = M == kAngle ? s.qnorm[q0 + q] : 0.f;
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int r = to + 16 * c;
                    float v = acc[i][c];
                    if (M == kAngle) {
                        v = v / (s.tnorm[sm.pos[r]] * qn);
                        if (v > 1.f) v = 1.f;
                        if (v >= th && r < nr) sw_emit<M, QI>(s, sm, q0, q, r, v);
                    } else if (v <= th && r < nr) {
                        sw_emit<M, QI>(s, sm, q0, q, r, v);
                    }
                }
            }
        } else {
            // the remaining pairs one by one: four in flight per warp
            constexpr int kP = 4;
            for (int p0 = warp * kP; p0 < n; p0 += (kSwThreads / 32) * kP) {
                float v[kP];
                const float *x[kP], *y[kP];
#pragma unroll
                for (int u = 0; u < kP; u++) {
                    const int e = sm.list[min(p0 + u, n - 1)];
                    x[u] = sm.rp[e & 127];
                    y[u] = qrow + (size_t)(e >> 7) * s.ld;
                    v[u] = 0.f;
                }
                if ((t.dim & 3) == 0) {
                    for (int k = lane * 4; k < t.dim; k += 128) {
                        float4 xa[kP], ya[kP];
#pragma unroll
                        for (int u = 0; u < kP; u++) {
                            xa[u] = __ldg(reinterpret_cast<const float4 *>(x[u] + k));
                            ya[u] = *reinterpret_cast<const float4 *>(y[u] + k);
                        }
#pragma unroll
                        for (int u = 0; u < kP; u++) {
                            v[u] = sw_term<M>(v[u], xa[u].x, ya[u].x);
                            v[u] = sw_term<M>(v[u], xa[u].y, ya[u].y);
                            v[u] = sw_term<M>(v[u], xa[u].z, ya[u].z);
                            v[u] = sw_term<M>(v[u], xa[u].w, ya[u].w);
                        }
                    }
                } else {
                    for (int k = lane; k < t.dim; k += 32)
#pragma unroll
                        for (int u = 0; u < kP; u++) v[u] = sw_term<M>(v[u], __ldg(x[u] + k), y[u][k]);
                }
#pragma unroll
                for (int u = 0; u < kP; u++) v[u] = M == kLinf ? warp_max(v[u]) : warp_sum(v[u]);
                float mine = 0.f;
#pragma unroll
                for (int u = 0; u < kP; u++)
                    if (lane == u) mine = v[u];
                if (lane < kP && p0 + lane < n) {
                    const int e = sm.list[p0 + lane];
                    if (mine <= sm.vthr[e >> 7]) sw_emit<M, QI>(s, sm, q0, e >> 7, e & 127, mine);
                }
            }
        }
        if (counts) {
            __syncthreads();
            if (tid < 16 * QI) {
                if (sm.cnt[tid]) atomicAdd(&s.cnt[q0 + tid], sm.cnt[tid]);
                if (sm.cnt2[tid]) atomicAdd(&s.cnt2[q0 + tid], sm.cnt2[tid]);
                sm.cnt[tid] = sm.cnt2[tid] = 0;
            }
        }
    }
    if (tid == 0 && s.a.stats && pairs) atomicAdd(&s.a.stats[0], pairs);
}

// ---------------------------------------------------------------- exact values

// The answers of one query from its candidate list, one CTA of 128 threads
// per sorted query.  kNN: candidates whose lower bound exceeds the k-th
// smallest upper bound are out, the rest get the reference's value and the k
// smallest (distance, id) are the answer.  Range counts add the listed
// objects within r to the certain ones.
__global__ void __launch_bounds__(128) k_sw_final(SweepArgs s)
{
    extern __shared__ __align__(16) unsigned char sw_smem[];
    FinalSmem &f = *reinterpret_cast<FinalSmem *>(sw_smem);
    const DevTree &t = s.a.t;
    const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = s.bq[i];
    const int mode = s.a.mode, k = s.a.k;
    int m = s.ccnt[i];
    int *cpos = s.cpos + (size_t)i * s.cap;
    float *cv = s.cv + (size_t)i * s.cap;
    const int self = s.self[i];
    if (m > s.cap) {
        // kNN: the listed candidates bound the k-th distance anew
        float R = 0.f;
        if (mode == kModeKnn) {
            for (int c = tid; c < s.cap; c += 128) {
                const float hi = cpos[c] == self ? 0.f
                                 : t.metric == kAngle ? (float)angle_of_cos_f64(cv[c]) * 1.00001f : sw_hi(t.metric, t.dim, cv[c]);
                f.key[c] = __float_as_uint(hi < FLT_MAX ? hi : FLT_MAX);
            }
            __syncthreads();
            R = __uint_as_float(cta_kth(f.key, s.cap, k, f.hist));
        }
        if (tid == 0) {
            const int at = atomicAdd(&s.ctr[1], 1);
            s.left[at] = make_int4(q, 0, 0, 0);
            s.left_R[at] = R;
            if (mode == kModeRangeCount || mode == kModeRangeTimed) {
                s.a.counts[q] = 0;   // the traversal adds to it
                if (mode == kModeRangeTimed) s.a.counts2[q] = 0;
            }
        }
        return;
    }
    const float *qrow = s.qrow + (size_t)i * s.ld;
    if (tid == 0) f.n = 0;
    __syncthreads();
    float B = FLT_MAX;
    if (mode == kModeKnn && t.metric != kAngle) {
        for (int c = tid; c < m; c += 128) f.key[c] = __float_as_uint(cpos[c] == self ? 0.f : sw_hi(t.metric, t.dim, cv[c]));
        __syncthreads();
        if (m > k) B = __uint_as_float(cta_kth(f.key, m, k, f.hist));
        for (int c = tid; c < m; c += 128)
            if (cpos[c] == self || sw_lo(t.metric, t.dim, cv[c]) <= B) f.pos[atomicAdd(&f.n, 1)] = cpos[c];
    } else if (t.metric == kAngle) {
        for (int c = tid; c < m; c += 128) {   // the value is exact already
            const double d = cpos[c] == self ? 0.0
                             : mode == kModeKnn ? angle_of_cos_f64(cv[c]) : (double)angle_of_cos_f32(cv[c]);
            if (mode == kModeKnn ? (d <= DBL_MAX) : ((float)d <= s.a.r)) {
                const int at = atomicAdd(&f.n, 1);
                f.d[at] = d;
                f.id[at] = t.id_list[cpos[c]];
            }
        }
    } else {
        for (int c = tid; c < m; c += 128) f.pos[c] = cpos[c];
        if (tid == 0) f.n = m;
    }
    __syncthreads();
    const int n = f.n;
    if (mode == kModeKnn && t.metric != kAngle) {
        exact_knn(f, t.metric, t.dim, t.trows, (size_t)t.dim, t.id_list, self, qrow, n, k);
        if (tid == 0 && s.a.stats) atomicAdd(&s.a.stats[2], (unsigned long long)n);
    } else if (mode != kModeKnn && t.metric != kAngle) {
        int wt = 0, wc = 0;
        // the staged terms lie over the warp's part of ts
        float(*ts)[33] = reinterpret_cast<float(*)[33]>(f.ts[warp]);
        for (int b0 = warp * kSwBatch; b0 < n; b0 += 4 * kSwBatch) {
            const int nb = min(kSwBatch, n - b0), p0 = f.pos[b0 + min(lane, nb - 1)];
            float d = range_batch<kSwBatch>(t.metric, t.dim, t.trows, (size_t)t.dim, p0, nb, qrow, ts, lane);
            if (lane < nb) {
                const int p = p0, id = t.id_list[p];
                if (p == self) d = 0.f;
                if (d <= s.a.r) {
                    if (mode == kModeRangeCount) {
                        wt++;
                    } else {
                        const int tq = s.a.qtime[q];
                        for (int e = s.a.ent_off[id], e1 = s.a.ent_off[id + 1]; e < e1; e++) {
                            const int4 v = s.a.ents[e];
                            wt += (v.x < tq && tq < v.y) ? 1 : 0;
                            wc += (v.z < tq && tq < v.w) ? 1 : 0;
                        }
                    }
                }
            }
        }
        if (tid == 0 && s.a.stats) atomicAdd(&s.a.stats[2], (unsigned long long)n);
        wt = __reduce_add_sync(0xffffffffu, wt);
        wc = __reduce_add_sync(0xffffffffu, wc);
        if (lane == 0) {
            if (wt) atomicAdd(&s.cnt[i], wt);
            if (wc) atomicAdd(&s.cnt2[i], wc);
        }
        __syncthreads();
    }
    if (tid == 0 && s.a.stats) atomicAdd(&s.a.stats[3], 1ull);
    if (mode == kModeRangeCount || mode == kModeRangeTimed) {
        if (tid == 0) {
            s.a.counts[q] = atomicAdd(&s.cnt[i], 0);
            if (mode == kModeRangeTimed) s.a.counts2[q] = atomicAdd(&s.cnt2[i], 0);
        }
        return;
    }
    if (t.metric == kAngle) sort_hits(f, n);
    for (int j = tid; j < k; j += 128) {
        const bool have = j < n;
        if (s.a.ids) s.a.ids[(size_t)q * k + j] = have ? f.id[j] : -1;
        if (s.a.dists) s.a.dists[(size_t)q * k + j] = have ? (float)f.d[j] : (float)t.infi_dis;
    }
    if (tid == 0) s.a.kth[q] = n >= k ? (float)f.d[k - 1] : (float)t.infi_dis;
}

// Range ids: the reference's values of the listed objects, in place of the
// filter's, kHitBatch rows per warp and one warp per CTA: hit numbers are
// uneven (58 on average, several hundred at most on 50,000 x 300), and idle
// warps of a larger CTA would hold registers that other queries' batches want
// (0.35 ms with eight warps, 0.37 with one CTA per query).
constexpr int kHitBatch = 16;
__global__ void __launch_bounds__(32) k_sw_hit_values(SweepArgs s)
{
    __shared__ float ts[kHitBatch][33];
    const DevTree &t = s.a.t;
    const int i = blockIdx.y, lane = threadIdx.x;
    const int m = s.ccnt[i], self = s.self[i];
    const int *cpos = s.cpos + (size_t)i * s.cap;
    float *cv = s.cv + (size_t)i * s.cap;
    const float *qrow = s.qrow + (size_t)i * s.ld;
    for (int b0 = blockIdx.x * kHitBatch; b0 < m; b0 += gridDim.x * kHitBatch) {
        const int nb = min(kHitBatch, m - b0);
        const int p = cpos[b0 + min(lane, nb - 1)];
        float d;
        if (t.metric == kAngle) d = angle_of_cos_f32(cv[b0 + min(lane, nb - 1)]);   // the value is exact already
        else d = range_batch<kHitBatch>(t.metric, t.dim, t.trows, (size_t)t.dim, p, nb, qrow, ts, lane);
        __syncwarp();
        if (lane < nb) cv[b0 + lane] = p == self ? 0.f : d;
    }
}

// Range ids: the listed objects within r, in (distance, id) order, back into
// the query's list as (id, value); their number to counts.  The keys sort as
// (float bits, id): the values are non-negative floats.
__global__ void __launch_bounds__(256) k_sw_hits(SweepArgs s)
{
    extern __shared__ __align__(16) unsigned char sw_smem[];
    __shared__ int hits;
    unsigned long long *key = reinterpret_cast<unsigned long long *>(sw_smem);
    const DevTree &t = s.a.t;
    const int i = blockIdx.x, tid = threadIdx.x;
    const int m = s.ccnt[i];
    int *cpos = s.cpos + (size_t)i * s.cap;
    float *cv = s.cv + (size_t)i * s.cap;
    if (tid == 0) hits = 0;
    __syncthreads();
    for (int c = tid; c < m; c += 256)
        if (cv[c] <= s.a.r)
            key[atomicAdd(&hits, 1)] = ((unsigned long long)__float_as_uint(cv[c]) << 32) | (unsigned)t.id_list[cpos[c]];
    __syncthreads();
    const int n = hits;
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    for (int c = n + tid; c < p2; c += 256) key[c] = ~0ull;
    __syncthreads();
    for (int size = 2; size <= p2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int c = tid; c < p2 / 2; c += 256) {
                const int lo = 2 * c - (c & (stride - 1)), hi = lo + stride;
                const unsigned long long x = key[lo], y = key[hi];
                if ((x > y) == ((lo & size) == 0)) {
                    key[lo] = y;
                    key[hi] = x;
                }
            }
            __syncthreads();
        }
    for (int c = tid; c < n; c += 256) {
        cpos[c] = (int)(uint32_t)key[c];
        cv[c] = __uint_as_float((uint32_t)(key[c] >> 32));
    }
    if (tid == 0) {
        s.a.counts[s.bq[i]] = n;
        if (s.a.stats) {
            atomicAdd(&s.a.stats[2], (unsigned long long)m);
            atomicAdd(&s.a.stats[3], 1ull);
        }
    }
}

__global__ void k_sw_longest(int n, const int *cnt, int *out)
{
    __shared__ int mx;
    if (threadIdx.x == 0) mx = 0;
    __syncthreads();
    int v = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v = max(v, cnt[i]);
    atomicMax(&mx, v);
    __syncthreads();
    if (threadIdx.x == 0) *out = mx;
}

inline int pow2_at_least(int n)
{
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// After a pass over a sample of the rows: the k-th smallest upper bound of the
// listed candidates where that is tighter than the query's bound; empty lists
// (the query object stays).
__global__ void __launch_bounds__(128) k_sw_tighten(SweepArgs s)
{
    __shared__ uint32_t key[kSwCap];
    __shared__ int hist[256];
    const DevTree &t = s.a.t;
    const int i = blockIdx.x, k = s.a.k, self = s.self[i];
    const int m = min(s.ccnt[i], s.cap);
    __syncthreads();
    if (threadIdx.x == 0) s.ccnt[i] = self >= 0 ? 1 : 0;
    if (m < k) return;
    for (int c = threadIdx.x; c < m; c += 128) {
        const int p = s.cpos[(size_t)i * s.cap + c];
        const float v = s.cv[(size_t)i * s.cap + c];
        const float hi = p == self ? 0.f : t.metric == kAngle ? (float)angle_of_cos_f64(v) * 1.00001f : sw_hi(t.metric, t.dim, v);
        key[c] = __float_as_uint(hi < FLT_MAX ? hi : FLT_MAX);
    }
    __syncthreads();
    const float R = __uint_as_float(cta_kth(key, m, k, hist));
    if (threadIdx.x == 0 && R < s.R[i]) {
        float vthr, vlow;
        sw_thresholds(t, R, true, vthr, vlow);
        s.R[i] = R;
        s.vthr[i] = vthr;
    }
}

// Buffers of a run of at most `tiles` query tiles; returns its bytes.
size_t plan_sweep(const gts_index *idx, int tiles, int qnum, unsigned char *base, SweepArgs *s, void **cub, size_t *cub_bytes)
{
    const int Qp = tiles * 128, ld = (idx->dim + kSwK - 1) / kSwK * kSwK;
    size_t off = 0, tb = 0;
    auto take = [&](size_t b) { size_t o = off; off += (b + 255) & ~(size_t)255; return base + o; };
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (int *)nullptr, (int *)nullptr, (int *)nullptr, (int *)nullptr, Qp, 0,
                                    32, (cudaStream_t)0);
    SweepArgs r{};
    r.Qp = Qp;
    r.ld = ld;
    r.left = (int4 *)take(sizeof(int4) * 2 * (size_t)qnum);   // two lists: this round's and the last one's
    r.left_R = (float *)take(4 * 2 * (size_t)qnum);
    r.cap = kSwCap;
    r.sample = 1;
    r.tq = 128;
    r.ctr = (int *)take(64);
    r.nrows = (int *)take(4 * (size_t)tiles);
    r.key = (int *)take(4 * (size_t)Qp * 5);   // key, sorted key, identity, order, batch query
    r.order = r.key + 3 * (size_t)Qp;
    r.bq = r.order + Qp;
    r.seed = (float *)take(4 * (size_t)Qp);
    r.qrow = (float *)take(4 * (size_t)Qp * ld);
    r.R = (float *)take(4 * (size_t)Qp * 4);
    r.vthr = r.R + Qp;
    r.vlow = r.vthr + Qp;
    r.qnorm = r.vlow + Qp;
    r.self = (int *)take(4 * (size_t)Qp * 4);
    r.ccnt = r.self + Qp;
    r.cnt = r.ccnt + Qp;
    r.cnt2 = r.cnt + Qp;
    r.dlo = (float *)take(4 * (size_t)std::max(idx->ncut_anc, 1) * Qp);
    r.dhi = (float *)take(4 * (size_t)std::max(idx->ncut_anc, 1) * Qp);
    r.rowpos = (int *)take(4 * (size_t)tiles * idx->num);
    r.cpos = (int *)take(4 * (size_t)Qp * kSwCap);
    r.cv = (float *)take(4 * (size_t)Qp * kSwCap);
    *cub = take(tb);
    *cub_bytes = tb;
    if (s) *s = r;
    return off;
}

template <int M, int QI>
int launch_tiles(gts_index *idx, SweepArgs s, bool sampled, cudaStream_t st)
{
    const int smem = (int)sizeof(SweepSmem<QI>);
    int per_sm = 1, dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    GTS_CUDA_TRY(cudaFuncSetAttribute(k_sw_pivots<M, QI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    GTS_CUDA_TRY(cudaFuncSetAttribute(k_sw_tile<M, QI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    GTS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sw_tile<M, QI>, kSwThreads, smem));
    const int tiles128 = s.ntiles;
    s.ntiles = (s.nq + 16 * QI - 1) / (16 * QI);
    if (s.nanc > 0) k_sw_pivots<M, QI><<<dim3((s.nanc + kSwRows - 1) / kSwRows, s.ntiles), kSwThreads, smem, st>>>(s);
    idx->kernel_launches += s.nanc > 0;
    // kNN seeds come from one neighbourhood of the tree order and are far off
    // for a few queries, which would then keep every row in play: a pass over
    // 1/16 of the rows first bounds every query by the whole data
    for (s.sample = sampled ? kSwSample : 1;; s.sample = 1) {
        sweep_cut_launch(s, tiles128, st);
        k_sw_tile<M, QI><<<nsm * std::max(per_sm, 1), kSwThreads, smem, st>>>(s);
        idx->kernel_launches += 2;
        if (s.sample == 1) break;
        k_sw_tighten<<<s.nq, 128, 0, st>>>(s);
        idx->kernel_launches++;
        GTS_CUDA_TRY(cudaMemsetAsync(s.ctr, 0, sizeof(int), st));
        GTS_CUDA_TRY(cudaMemsetAsync(s.nrows, 0, sizeof(int) * tiles128, st));
    }
    GTS_CUDA_TRY(cudaGetLastError());
    return GTS_OK;
}

template <int QI>
int launch_metric(gts_index *idx, const SweepArgs &s, bool sampled, cudaStream_t st)
{
    switch (idx->metric) {
    case kL2: return launch_tiles<kL2, QI>(idx, s, sampled, st);
    case kL1: return launch_tiles<kL1, QI>(idx, s, sampled, st);
    case kLinf: return launch_tiles<kLinf, QI>(idx, s, sampled, st);
    default: return launch_tiles<kAngle, QI>(idx, s, sampled, st);
    }
}

// The ordered hits of the run's queries [q0, q1) into call order; offsets of
// the run's queries, of which q0's first hit is number `base`.
__global__ void k_sw_copy_hits(SweepArgs s, int q0, int q1, int base)
{
    const int i = blockIdx.x;
    const int q = s.bq[i];
    if (q < q0 || q >= q1) return;
    const int n = s.a.counts[q], o = s.a.offsets[q - s.q0] - base;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        s.a.rids[o + c] = s.cpos[(size_t)i * s.cap + c];
        s.a.rdists[o + c] = s.cv[(size_t)i * s.cap + c];
    }
}

}  // namespace

void sweep_cut_launch(const SweepArgs &s, int ntiles, cudaStream_t st)
{
    k_sw_cut<<<dim3((s.ncut + 255) / 256, ntiles), 256, 0, st>>>(s);
}

// The sizes from which on the sweep is the sooner one.  A batch of one tile
// waits for a chain of stages of 16 dimensions, 2.9 us each for the pivots and
// 5.2 for the rows (1.1 and 2.2 with the tile of 32 queries).  A CTA of the traversal
// waits for its query's objects, some 18 ns each, and for a second wave from
// about 256 queries on; L2 kNN values and angles cost it more per dimension.
// Traversal and sweep, us, a batch of 100 where not given:
//   L1 range  1,000 x 1,000  177  775    4,000 x 128  143  183    5,000 x 64  241  159
//     2,000 x 33, 1,000 queries  275  155    2,000 x 300, 30 queries  131  178
//   L1 kNN    2,000 x 300    213  348    4,000 x 300  299  345    4,000 x 128, 300 queries  497  252
//   L2 range  2,000 x 300    249  317    4,000 x 300  318  342    60,000 x 300  2,649  223
//   L2 kNN      500 x 1,000 1,795 827
//   angle     2,000 x 33     101  132    1,000 x 300  191  251    4,000 x 64  251  183
// Objects exactly equal to the query lie in a leaf or two of a deep tree: 0.43 ms
// for 10,000 queries over 1,000,000 x 128, 0.88 by the sweep.
static bool sweep_pays(const gts_index *idx, const SearchArgs &a)
{
    const long long n = idx->num, d = idx->dim, q = a.qnum;
    if (n * d < 1 << 16 && n * q < 1 << 20) return false;
    const bool knn = a.mode == kModeKnn, few = q <= kSwFew;
    const long long waves = n * std::max(q, 256ll) / 256;   // objects in the traversal's way
    if (knn && idx->metric == kL2) return true;
    if (a.mode == kModeRangeIds) return n >= 4 * d;         // two traversals and a sort on the host
    if (!knn && a.r == 0.f && n <= 32ll * idx->nleaf) return false;
    if (idx->metric == kAngle) return few ? n * d >= 1 << 17 : waves >= 4096 || (waves >= 2000 && n * d >= 250000);
    if (idx->metric == kL2) return few ? n >= 2 * d : waves >= 2048 && waves >= 8 * d;
    return few ? n >= 2048 && (knn || n >= 16 * d) : waves >= 4096 && waves >= (knn ? 8 : 48) * d;
}

// Batches the sweep takes: row metrics of more dimensions than a lane filters
// alone, without deletions, learned seeds, or a caller's choice of the
// traversal (pinned threads, a set hand-over threshold); radii whose squares
// stay finite.
bool sweep_takes(const gts_index *idx, const SearchArgs &a)
{
    if (idx->metric == kEdit || idx->dim <= kLaneRowDim || idx->dim > 2048 || idx->ncut < 1) return false;
    if (a.deleted || a.seed_r2_bits || a.items_in || a.qstrs) return false;
    const int slot = a.mode == kModeRangeTimed ? kModeRangeCount : a.mode;
    if (idx->plain_pinned[slot] || (a.mode != kModeKnn && idx->plain_split_set)) return false;
    if (a.mode == kModeKnn ? a.k > 128 : !(a.r >= 0.f && a.r <= 1e15f)) return false;
    return sweep_pays(idx, a);
}

namespace {

// A batch's buffers and run size within the call's budget; false when the
// batch is not one for the sweep.
struct SweepBatch {
    SweepArgs s;
    size_t bytes = 0;
    void *cub = nullptr;
    size_t cub_bytes = 0;
    int run = 0;   // queries per run
};

bool sweep_begin(gts_index *idx, const SearchArgs &a, SweepBatch *b)
{
    if (!sweep_takes(idx, a)) return false;
    const size_t budget = search_budget(idx);
    int tiles = std::min(kSwMaxTiles, (a.qnum + 127) / 128);
    size_t bytes;
    for (;;) {
        bytes = plan_sweep(idx, tiles, a.qnum, nullptr, nullptr, &b->cub, &b->cub_bytes);
        if (bytes <= budget || tiles == 1) break;
        tiles = (tiles + 1) / 2;
    }
    if (bytes > budget || ensure_scratch(idx, bytes) != GTS_OK) return false;
    plan_sweep(idx, tiles, a.qnum, (unsigned char *)idx->scratch, &b->s, &b->cub, &b->cub_bytes);
    b->run = tiles * 128;
    b->bytes = bytes;
    b->s.a = a;
    b->s.cut = idx->cut_node;
    b->s.ncut = idx->ncut;
    b->s.anc = idx->cut_anc;
    b->s.nanc = idx->ncut_anc;
    b->s.anc_idx = idx->cut_anc_idx;
    b->s.tnorm = idx->tnorm;
    return true;
}

// Ring bounds, filter and answers of the run's queries, once their places and
// bounds are known.
int sweep_pass(gts_index *idx, SweepArgs &s, cudaStream_t st)
{
    k_sw_query<<<(s.Qp + 7) / 8, 256, 0, st>>>(s);
    // 32 queries per tile when there are no more of them: the 128-wide tile
    // would multiply padding
    const bool sampled = s.a.mode == kModeKnn && !s.again && idx->num >= kSwSampleMin;
    int rc = s.nq <= kSwFew ? launch_metric<2>(idx, s, sampled, st) : launch_metric<8>(idx, s, sampled, st);
    if (rc) return rc;
    idx->kernel_launches++;
    return GTS_OK;
}

int sweep_answers(gts_index *idx, SweepArgs &s, cudaStream_t st)
{
    GTS_CUDA_TRY(cudaFuncSetAttribute(k_sw_final, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinalSmem)));
    k_sw_final<<<s.nq, 128, sizeof(FinalSmem), st>>>(s);
    idx->kernel_launches++;
    GTS_CUDA_TRY(cudaGetLastError());
    return GTS_OK;
}

// One run of the batch's queries from q0: seeds and order, then the pass.
int sweep_enqueue(gts_index *idx, SweepBatch &b, int q0, cudaStream_t st)
{
    SweepArgs &s = b.s;
    int key_bits = 1;
    while (key_bits < 31 && (1 << key_bits) < idx->num) key_bits++;
    s.q0 = q0;
    s.nq = std::min(b.run, s.a.qnum - q0);
    s.ntiles = (s.nq + 127) / 128;
    int *skey = s.key + s.Qp, *iota = skey + s.Qp;
    if (s.nq > 128 || s.a.mode == kModeKnn) {   // a tile of range queries needs neither places nor seeds
        k_sw_seed<<<s.nq, kSwThreads, sizeof(float) * (size_t)idx->dim, st>>>(s, kSwWindow);
        idx->kernel_launches++;
    }
    if (s.nq > 128) {   // queries of one tile should be neighbours in the tree order
        k_sw_iota<<<(s.nq + 255) / 256, 256, 0, st>>>(s.nq, iota);
        idx->kernel_launches++;
        GTS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(b.cub, b.cub_bytes, s.key, skey, iota, s.order, s.nq, 0, key_bits,
                                                     st));
    }
    return sweep_pass(idx, s, st);
}

// Queries left to the traversal, and whether every query id was in range.
int sweep_outcome(gts_index *idx, const SweepBatch &b, int *left, bool *ok, cudaStream_t st)
{
    int h[2] = {0, 0}, status = 0;
    GTS_CUDA_TRY(cudaMemcpyAsync(h, b.s.ctr, sizeof(h), cudaMemcpyDeviceToHost, st));
    GTS_CUDA_TRY(cudaMemcpyAsync(&status, idx->d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    GTS_CUDA_TRY(cudaStreamSynchronize(st));
    *left = h[1];
    *ok = status == 0;
    return GTS_OK;
}

}  // namespace

int run_sweep(gts_index *idx, const SearchArgs &a, cudaStream_t st, int *done, const int4 **items, int *n_left)
{
    *done = 0;
    *n_left = 0;
    if (idx->metric == kEdit) return run_sweep_edit(idx, a, st, done, items, n_left);
    SweepBatch b;
    if (!sweep_begin(idx, a, &b)) return GTS_OK;
    int rc;
    GTS_CUDA_TRY(cudaMemsetAsync(b.s.ctr, 0, 64, st));
    for (int q0 = 0; q0 < a.qnum; q0 += b.run)
        if ((rc = sweep_enqueue(idx, b, q0, st)) || (rc = sweep_answers(idx, b.s, st))) return rc;
    bool ok = false;
    if ((rc = sweep_outcome(idx, b, n_left, &ok, st))) return rc;
    // a kNN query whose seed let too many objects in has a better bound now
    int4 *const lists[2] = {b.s.left, b.s.left + a.qnum};
    float *const bounds[2] = {b.s.left_R, b.s.left_R + a.qnum};
    int cur = 0;
    for (int round = 0; round < kSwRounds && ok && a.mode == kModeKnn && *n_left > 0; round++) {
        SweepArgs &s = b.s;
        const int n = *n_left;
        s.again = lists[cur];
        s.again_R = bounds[cur];
        cur ^= 1;
        s.left = lists[cur];
        s.left_R = bounds[cur];
        GTS_CUDA_TRY(cudaMemsetAsync(s.ctr, 0, 64, st));
        for (int q0 = 0; q0 < n; q0 += b.run) {
            s.q0 = q0;
            s.nq = std::min(b.run, n - q0);
            s.ntiles = (s.nq + 127) / 128;
            if ((rc = sweep_pass(idx, s, st)) || (rc = sweep_answers(idx, s, st))) return rc;
        }
        if ((rc = sweep_outcome(idx, b, n_left, &ok, st))) return rc;
    }
    if (!ok) {   // a query id out of range: the traversal reports it
        GTS_CUDA_TRY(cudaMemsetAsync(idx->d_status, 0, sizeof(int), st));
        return GTS_OK;
    }
    *done = 1;
    *items = b.s.left;
    return GTS_OK;
}

int sweep_range_ids(gts_index *idx, const int *d_qids, int qnum, float r, int *d_counts, int *counts_out,
                    int *offsets_out, int *ids_out, float *dists_out, size_t capacity, size_t *total, int *done,
                    cudaStream_t st)
{
    *done = 0;
    *total = 0;
    SearchArgs a{};
    a.qids = d_qids;
    a.qnum = qnum;
    a.mode = kModeRangeIds;
    a.r = r;
    a.counts = d_counts;
    fill_search_args(idx, a);
    SweepBatch b;
    if (!sweep_begin(idx, a, &b)) return GTS_OK;
    GTS_CUDA_TRY(cudaMemsetAsync(idx->d_status, 0, sizeof(int), st));
    GTS_CUDA_TRY(cudaMemsetAsync(idx->d_stats, 0, kStatsN * sizeof(unsigned long long), st));
    struct Lists {   // longer lists than the run's own, freed on every way out
        void *p = nullptr;
        ~Lists() { if (p) dev_free(p); }
    } lists;
    int rc;
    GTS_CUDA_TRY(cudaMemsetAsync(b.s.ctr, 0, 64, st));
    for (int q0 = 0; q0 < qnum; q0 += b.run) {
        if ((rc = sweep_enqueue(idx, b, q0, st))) return rc;
        const int nq = b.s.nq;
        // the lists are counted in full: make room for the longest and go
        // over the rows again when it did not fit
        int longest = 0;
        bool ok = false;
        k_sw_longest<<<1, 256, 0, st>>>(nq, b.s.ccnt, b.s.ctr + 1);
        if ((rc = sweep_outcome(idx, b, &longest, &ok, st))) return rc;
        if (!ok || longest > kSwHitCap) return GTS_OK;
        if (longest > b.s.cap) {
            const size_t list = sizeof(int) * (size_t)b.s.Qp * longest;
            if (b.bytes + 2 * list > search_budget(idx)) return GTS_OK;
            void *buf = nullptr;
            if (lists.p) dev_free(lists.p);
            lists.p = nullptr;
            if (dev_malloc(&buf, 2 * list) != cudaSuccess) {
                cudaGetLastError();
                return GTS_OK;
            }
            lists.p = buf;
            b.s.cap = longest;
            b.s.cpos = (int *)buf;
            b.s.cv = (float *)((unsigned char *)buf + list);
            if ((rc = sweep_pass(idx, b.s, st))) return rc;
        }
        k_sw_hit_values<<<dim3(std::min(64, (longest + kHitBatch - 1) / kHitBatch), nq), 32, 0, st>>>(b.s);
        const size_t hsm = sizeof(unsigned long long) * (size_t)pow2_at_least(longest);
        GTS_CUDA_TRY(cudaFuncSetAttribute(k_sw_hits, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hsm));
        k_sw_hits<<<nq, 256, hsm, st>>>(b.s);
        idx->kernel_launches += 3;
        GTS_CUDA_TRY(cudaGetLastError());
        GTS_CUDA_TRY(cudaMemcpyAsync(counts_out + q0, d_counts + q0, sizeof(int) * nq, cudaMemcpyDeviceToHost, st));
        GTS_CUDA_TRY(cudaStreamSynchronize(st));
        const size_t base = *total;
        for (int i = q0; i < q0 + nq; i++) {
            offsets_out[i] = (int)*total;
            *total += (size_t)counts_out[i];
        }
        if (*total > capacity || *total > 0x7fffffff || *total == base) continue;
        // the run's hits, from the lists into call order and out, as many
        // queries at a time as the call's budget has room for
        const size_t used = b.bytes + (lists.p ? 2 * sizeof(int) * (size_t)b.s.Qp * b.s.cap : 0);
        const size_t room = search_budget(idx) > used ? search_budget(idx) - used : 0;
        const size_t ob = (sizeof(int) * (size_t)nq + 255) & ~(size_t)255;
        for (int i0 = q0, i1; i0 < q0 + nq; i0 = i1) {
            auto bytes_to = [&](int i) {   // of the hits of queries i0 .. i
                const size_t n = (size_t)offsets_out[i] + counts_out[i] - offsets_out[i0];
                return ob + 2 * ((4 * n + 255) & ~(size_t)255);
            };
            if (bytes_to(i0) > room) return GTS_OK;
            for (i1 = i0 + 1; i1 < q0 + nq && bytes_to(i1) <= room; i1++) {}
            const size_t need = bytes_to(i1 - 1), nb = (need - ob) / 2;
            const size_t first = (size_t)offsets_out[i0], n = (size_t)offsets_out[i1 - 1] + counts_out[i1 - 1] - first;
            if (n == 0) continue;
            void *buf = nullptr;
            if ((rc = ensure_hits(idx, need, room, &buf))) return rc;
            int *d_off = (int *)buf, *d_hid = (int *)((unsigned char *)buf + ob);
            float *d_hd = (float *)((unsigned char *)buf + ob + nb);
            GTS_CUDA_TRY(cudaMemcpyAsync(d_off, offsets_out + q0, sizeof(int) * nq, cudaMemcpyHostToDevice, st));
            b.s.a.offsets = d_off;
            b.s.a.rids = d_hid;
            b.s.a.rdists = d_hd;
            k_sw_copy_hits<<<nq, 64, 0, st>>>(b.s, i0, i1, (int)first);
            idx->kernel_launches++;
            GTS_CUDA_TRY(cudaGetLastError());
            if (ids_out) GTS_CUDA_TRY(cudaMemcpyAsync(ids_out + first, d_hid, 4 * n, cudaMemcpyDeviceToHost, st));
            if (dists_out) GTS_CUDA_TRY(cudaMemcpyAsync(dists_out + first, d_hd, 4 * n, cudaMemcpyDeviceToHost, st));
            GTS_CUDA_TRY(cudaStreamSynchronize(st));
        }
    }
    *done = 1;
    return GTS_OK;
}

}  // namespace gts
