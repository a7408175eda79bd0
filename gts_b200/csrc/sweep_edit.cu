// sweep_edit.cu -- the batched sweep of the plain form for strings.
//
// As sweep.cu, with 32 queries per tile: the ring bounds keep the cut nodes
// that some query of the tile can reach, and every object of those is tested
// against the tile's queries.  The traversal spent 166 ms on 10,000 range-2
// queries over 1,000,000 words (8.8 here): a leaf of ten strings keeps few of a
// CTA's threads busy and every query reads the signatures and strings it reaches
// for itself.  Here
//
//   * a thread holds one object's character counts (metric.cuh, str_sig) in
//     registers and tests them against the 32 queries' in shared memory: the
//     length and count bounds leave about 5% of the pairs at radius 2;
//   * the surviving pairs of a row tile are listed and spread over the CTA's
//     threads, which run the bit-parallel edit distance in 32-bit words (the
//     query is the pattern, its character masks in shared memory, the object's
//     first 32 characters beside them) and stop once the remaining characters
//     cannot bring the distance within the bound.
//
// Distances are whole numbers, so kNN keeps a histogram of the distances found
// per query: its k-th entry is the running bound, and after the sweep the
// exact k-th distance.  Queries are taken in the order of their lengths, then
// of their places in the tree: a tile then needs few lengths of strings, and
// leaves out the rest when it lists its rows.  Queries of 33 to 64 characters
// get a pass of their own in 64-bit words, or take the others along where many
// strings are that long; longer ones, and queries whose list cannot hold their
// candidates, go to the traversal.
#include <cub/device/device_radix_sort.cuh>
#include <algorithm>
#include <climits>
#include "sweep.cuh"

namespace gts {

namespace {

constexpr int kSeThreads = 256;
constexpr int kSeTq = 32;              // queries per tile
constexpr int kSeMaxTiles = 64;        // query tiles per run
constexpr int kSeRows = 256;           // rows per row tile, one per thread
constexpr int kSeChunk = 8;            // row tiles per work item
constexpr int kSeWindow = 1024;        // objects around a query's place that bound its k-th distance
constexpr int kSeCap = 2048;           // candidates listed per query
constexpr int kSeHist = 128;           // distances are at most 108
constexpr int kSeRounds = 2;           // further passes, in 64-bit words
constexpr int kSeTextLd = kPackChars / 4 + 1;   // words per row's characters in shared memory (odd: no bank conflicts)

struct EditArgs {
    SweepArgs s;
    int wide;               // the pass takes patterns of up to 64 characters (else 32)
    uint4 *lens_ok;         // per tile: lengths within some query's radius
    const uint4 *tpack;
    int *qlen;              // [Qp] pattern length; -1: not swept
    uint32_t *qpack;        // [Qp][16] first 64 characters
    uint32_t *qsig;         // [Qp][8] low and high nibbles of the signature
    int *hist;              // kNN: [Qp][kSeHist] distances found
};

// One step of the bit-parallel column (Myers 1999, Hyyro's formulation) on a
// 32- or 64-bit word, as edit_myers64.
template <typename W>
struct Myers {
    W pv, mv, hi;
    int score;
    __device__ __forceinline__ void start(int m)
    {
        pv = ~(W)0;
        mv = 0;
        hi = (W)1 << (m - 1);
        score = m;
    }
    __device__ __forceinline__ void step(W eq)
    {
        const W xv = eq | mv;
        const W xh = (((eq & pv) + pv) ^ pv) | eq;
        W ph = mv | ~(xh | pv), mh = pv & xh;
        score += (ph & hi) ? 1 : ((mh & hi) ? -1 : 0);
        ph = (ph << 1) | (W)1;
        mh <<= 1;
        pv = mh | ~(xv | ph);
        mv = ph & xv;
    }
};

// Edit distance of the pattern behind peq (m characters, at most the word's
// bits) to a text of n characters, its first kPackChars from words, the rest
// from tail; some value above limit where the distance is above limit.
template <typename W>
__device__ __forceinline__ int edit_words(const W *peq, int m, const uint32_t *words, const char *tail, int n, int limit)
{
    if (m == 0) return n;
    if (n == 0) return m;
    Myers<W> d;
    d.start(m);
    for (int j0 = 0; j0 < n; j0 += 4) {
        uint32_t w;
        if (j0 < kPackChars) {
            w = words[j0 >> 2];
        } else {
            w = 0;
            for (int u = 0; u < 4 && j0 + u < n; u++) w |= (uint32_t)(unsigned char)tail[j0 + u] << (8 * u);
        }
        const int e = min(4, n - j0);
        for (int u = 0; u < e; u++) {
            d.step(peq[w & 255u]);
            w >>= 8;
        }
        if (d.score - (n - j0 - e) > limit) return INT_MAX;   // a character lowers it by one at most
    }
    return d.score;
}

__device__ __forceinline__ int str_len(int n) { return min(max(n, 0), kStrStride); }

__device__ __forceinline__ void set_bit(uint32_t *p, int i) { atomicOr(p, 1u << i); }
__device__ __forceinline__ void set_bit(unsigned long long *p, int i) { atomicOr(p, 1ull << i); }

// ---------------------------------------------------------------- seeds

// The masks of one query's characters, made by the CTA.
template <typename W>
__device__ __forceinline__ void make_peq(W *peq, const char *src, int m)
{
    for (int c = threadIdx.x; c < 256; c += blockDim.x) peq[c] = 0;
    __syncthreads();
    if ((int)threadIdx.x < m) set_bit(&peq[(unsigned char)src[threadIdx.x]], threadIdx.x);
    __syncthreads();
}

template <typename W>
__device__ __forceinline__ int edit_to_id(const DevTree &t, const W *peq, int m, int id)
{
    const char *txt = t.strs + (size_t)id * kStrStride;
    const int n = str_len(t.lens[id]);
    if (m == 0) return n;
    if (n == 0) return m;
    Myers<W> d;
    d.start(m);
    for (int j = 0; j < n; j++) d.step(peq[(unsigned char)txt[j]]);
    return d.score;
}

// One CTA per query of the batch: its sort key (length, then its place in the
// tree order), and for kNN the k-th smallest distance over the kSeWindow
// objects around that place.
__global__ void __launch_bounds__(kSeThreads) k_se_seed(EditArgs e, int pos_bits)
{
    __shared__ unsigned long long peq[256];
    __shared__ int hist[kSeHist];
    __shared__ int s_node;
    const SweepArgs &s = e.s;
    const DevTree &t = s.a.t;
    const int q = blockIdx.x, tid = threadIdx.x;
    const bool by_data = s.a.qstrs != nullptr, knn = s.a.mode == kModeKnn;
    const int qid = by_data ? -1 : s.a.qids[q];
    if (!by_data && (qid < 0 || qid >= t.num)) {
        if (tid == 0) {
            atomicMax(s.a.status, (int)kKsBadQuery);
            s.key[q] = 0;
            s.seed[q] = -1.f;
        }
        return;
    }
    const char *src = by_data ? s.a.qstrs + (size_t)q * kStrStride : t.strs + (size_t)qid * kStrStride;
    const int m = min(max(by_data ? s.a.qlens[q] : t.lens[qid], 0), kStrStride - 1);
    int pos = by_data ? 0 : t.pos_of_id[qid];
    const int pos_shift = max(0, pos_bits - 24);   // 7 bits of length, up to 24 of position
    if ((!by_data && !knn) || m > 64) {
        if (tid == 0) {
            s.key[q] = m << 24 | pos >> pos_shift;
            s.seed[q] = -1.f;
        }
        return;
    }
    make_peq(peq, src, m);
    if (by_data) {   // down the rings its pivot distances fall into
        int node = 0;
        while (t.node_pivot[node] >= 0) {
            if (tid == 0) {
                const float d = (float)edit_to_id(t, peq, m, t.node_pivot[node]);
                int at = -1;
                for (int i = 0; i < t.order; i++) {
                    const long c = (long)node * t.order + i + 1;
                    if (c >= t.max_node_num || !(t.node_flags[c] & kExists) || t.node_size[c] == 0) continue;
                    if (at < 0 || t.node_min_dis[c] <= d) at = (int)c;
                }
                s_node = at;
            }
            __syncthreads();
            const int next = s_node;
            __syncthreads();
            if (next < 0) break;
            node = next;
        }
        pos = min(t.node_lid[node] + t.node_size[node] / 2, t.num - 1);
    }
    if (tid == 0) s.key[q] = m << 24 | pos >> pos_shift;
    if (!knn) return;
    for (int i = tid; i < kSeHist; i += kSeThreads) hist[i] = 0;
    __syncthreads();
    const int w = min(kSeWindow, t.num), w0 = max(0, min(pos - w / 2, t.num - w));
    for (int i = tid; i < w; i += kSeThreads) {
        const int p = w0 + i;
        const uint4 a = e.tpack[2 * (size_t)p], b = e.tpack[2 * (size_t)p + 1];
        const uint32_t words[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        const int d = edit_words(peq, m, words, t.tstrs + (size_t)p * kStrStride, str_len(t.tlens[p]), INT_MAX);
        atomicAdd(&hist[min(d, kSeHist - 1)], 1);
    }
    __syncthreads();
    if (tid == 0) {
        int R = kSeHist - 1, run = 0;
        for (int d = 0; d < kSeHist; d++) {
            run += hist[d];
            if (run >= s.a.k) {
                R = d;
                break;
            }
        }
        s.seed[q] = (float)R;
        if (s.a.stats) atomicAdd(&s.a.stats[0], (unsigned long long)w);
    }
}

__global__ void k_se_iota(int n, int *v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}

// One thread per sorted query slot: its pattern, signature and radius, empty
// lists.  A query the pass does not take goes to the next one's list, and
// past the last pass to the traversal.  A warp is a tile: it also makes the
// tile's mask of string lengths.
__global__ void __launch_bounds__(128) k_se_query(EditArgs e)
{
    const SweepArgs &s = e.s;
    const DevTree &t = s.a.t;
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (blockIdx.x == 0) {   // the pass's counters
        for (int j = threadIdx.x; j < s.ntiles; j += 128) s.nrows[j] = 0;
        if (threadIdx.x == 0) s.ctr[0] = 0;
    }
    if (i >= s.Qp) return;
    const bool have = i < s.nq;
    const int q = !have ? -1 : (s.again ? s.again[s.q0 + i].x : s.order[s.q0 + i]);
    s.bq[i] = q;
    s.ccnt[i] = s.cnt[i] = s.cnt2[i] = 0;
    float R = -1.f;
    int m = -1;
    const int qid = have && !s.a.qstrs ? s.a.qids[q] : -1;
    if (have && (s.a.qstrs || (qid >= 0 && qid < t.num))) {
        const char *src = s.a.qstrs ? s.a.qstrs + (size_t)q * kStrStride : t.strs + (size_t)qid * kStrStride;
        m = min(max(s.a.qstrs ? s.a.qlens[q] : t.lens[qid], 0), kStrStride - 1);
        if (m > (e.wide ? 64 : 32)) {
            const int at = atomicAdd(&s.ctr[1], 1);
            s.left[at] = make_int4(q, 0, 0, 0);
            s.left_R[at] = s.seed[q];
            m = -1;
            if (s.a.mode != kModeKnn) {
                s.a.counts[q] = 0;   // the traversal adds to it
                if (s.a.mode == kModeRangeTimed) s.a.counts2[q] = 0;
            }
        } else {
            R = s.a.mode != kModeKnn ? floorf(fminf(s.a.r, (float)(kSeHist - 1)))
                                     : (s.again ? s.again_R[s.q0 + i] : s.seed[q]);
            const uint4 g = str_sig(src, m);
            const uint32_t w[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                e.qsig[8 * (size_t)i + c] = w[c] & 0x0F0F0F0Fu;
                e.qsig[8 * (size_t)i + 4 + c] = (w[c] >> 4) & 0x0F0F0F0Fu;
            }
            for (int c = 0; c < 16; c++) {
                uint32_t v = 0;
                for (int u = 0; u < 4; u++)
                    if (4 * c + u < m) v |= (uint32_t)(unsigned char)src[4 * c + u] << (8 * u);
                e.qpack[16 * (size_t)i + c] = v;
            }
        }
    }
    s.R[i] = R;
    e.qlen[i] = m;
    uint32_t ok[4] = {0, 0, 0, 0};
    if (m >= 0 && R >= 0.f)
        for (int n = max(0, m - (int)R); n <= min(127, m + (int)R); n++) ok[n >> 5] |= 1u << (n & 31);
#pragma unroll
    for (int c = 0; c < 4; c++) ok[c] = __reduce_or_sync(0xffffffffu, ok[c]);
    if ((i & 31) == 0) e.lens_ok[i / kSeTq] = make_uint4(ok[0], ok[1], ok[2], ok[3]);
    if (s.a.mode == kModeKnn)
        for (int d = 0; d < kSeHist; d++) e.hist[(size_t)i * kSeHist + d] = 0;
}

// Distances of one query per CTA to the cut nodes' ancestors' pivots.
template <typename W>
__global__ void __launch_bounds__(kSeThreads) k_se_pivots(EditArgs e)
{
    __shared__ W peq[256];
    const SweepArgs &s = e.s;
    const DevTree &t = s.a.t;
    const int i = blockIdx.x, m = e.qlen[i];
    if (m < 0) return;
    make_peq(peq, reinterpret_cast<const char *>(e.qpack + 16 * (size_t)i), m);
    for (int a = blockIdx.y * kSeThreads + threadIdx.x; a < s.nanc; a += gridDim.y * kSeThreads) {
        const float d = (float)edit_to_id(t, peq, m, t.node_pivot[s.anc[a]]);
        s.dlo[(size_t)a * s.Qp + i] = d;
        s.dhi[(size_t)a * s.Qp + i] = d;
    }
}

// ---------------------------------------------------------------- tiles

template <typename W>
struct EditSmem {
    W peq[kSeTq][256];
    uint32_t text[kSeRows * kSeTextLd];
    uint32_t sig[kSeTq][8];
    int pos[kSeRows], len[kSeRows];
    unsigned short list[kSeRows * kSeTq];   // query << 8 | row
    int qlen[kSeTq], R[kSeTq], cnt[kSeTq], cnt2[kSeTq];
    int wsum[kSeThreads / 32];
    int item, nlist;
};

// Persistent CTAs take (query tile, chunk of row tiles) items, query tiles
// outermost: the tile's masks stay while the CTA goes over its rows.
template <typename W>
__global__ void __launch_bounds__(kSeThreads, sizeof(W) == 4 ? 3 : 2) k_se_tile(EditArgs e)
{
    extern __shared__ __align__(16) unsigned char se_smem[];
    EditSmem<W> &sm = *reinterpret_cast<EditSmem<W> *>(se_smem);
    const SweepArgs &s = e.s;
    const DevTree &t = s.a.t;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int mode = s.a.mode;
    int maxc = 0;   // chunks of the longest row list
    for (int i = 0; i < s.ntiles; i++) maxc = max(maxc, (s.nrows[i] + kSeRows * kSeChunk - 1) / (kSeRows * kSeChunk));
    int cur = -1;
    unsigned long long tested = 0, exact = 0;
    for (;;) {
        __syncthreads();
        if (tid == 0) sm.item = atomicAdd(&s.ctr[0], 1);
        __syncthreads();
        const int tile = maxc > 0 ? sm.item / maxc : s.ntiles, ch = sm.item - tile * maxc;
        if (tile >= s.ntiles) break;
        const int nr = s.nrows[tile], r0 = ch * kSeRows * kSeChunk;
        if (r0 >= nr) continue;
        const int q0 = tile * kSeTq;
        if (tile != cur) {
            for (int i = tid; i < kSeTq * 256; i += kSeThreads) (&sm.peq[0][0])[i] = 0;
            sm.sig[tid >> 3][tid & 7] = e.qsig[8 * (size_t)q0 + tid];
            if (tid < kSeTq) {
                sm.qlen[tid] = e.qlen[q0 + tid];
                sm.cnt[tid] = sm.cnt2[tid] = 0;
                sm.R[tid] = (int)s.R[q0 + tid];
            }
            __syncthreads();
            constexpr int kBits = 8 * (int)sizeof(W);
            for (int i = tid; i < kSeTq * kBits; i += kSeThreads) {
                const int q = i / kBits, j = i % kBits;
                if (j < sm.qlen[q])
                    set_bit(&sm.peq[q][(e.qpack[16 * (size_t)(q0 + q) + (j >> 2)] >> (8 * (j & 3))) & 255u], j);
            }
            cur = tile;
        }
        for (int rt = r0; rt < min(nr, r0 + kSeRows * kSeChunk); rt += kSeRows) {
            __syncthreads();   // the last row tile's pairs are done
            if (mode == kModeKnn && tid < kSeTq && sm.R[tid] > 0) {
                // the running bound: the k-th distance found so far
                const volatile int *h = e.hist + (size_t)(q0 + tid) * kSeHist;
                int run = 0;
                for (int d = 0; d < sm.R[tid]; d++) {
                    run += h[d];
                    if (run >= s.a.k) {
                        sm.R[tid] = d;
                        break;
                    }
                }
            }
            const int n = min(kSeRows, nr - rt);
            const int p = s.rowpos[(size_t)tile * t.num + rt + min(tid, n - 1)];
            const uint4 g = t.tsig[p];
            const int len = str_len(t.tlens[p]);
            const uint4 a = e.tpack[2 * (size_t)p], b = e.tpack[2 * (size_t)p + 1];
            uint32_t *tx = sm.text + tid * kSeTextLd;
            tx[0] = a.x; tx[1] = a.y; tx[2] = a.z; tx[3] = a.w;
            tx[4] = b.x; tx[5] = b.y; tx[6] = b.z; tx[7] = b.w;
            sm.pos[tid] = p;
            sm.len[tid] = len;
            __syncthreads();
            const uint32_t w[8] = {g.x & 0x0F0F0F0Fu, g.y & 0x0F0F0F0Fu, g.z & 0x0F0F0F0Fu, g.w & 0x0F0F0F0Fu,
                                   (g.x >> 4) & 0x0F0F0F0Fu, (g.y >> 4) & 0x0F0F0F0Fu, (g.z >> 4) & 0x0F0F0F0Fu,
                                   (g.w >> 4) & 0x0F0F0F0Fu};
            uint32_t pass = 0;   // queries whose bounds admit this object
#pragma unroll 8
            for (int q = 0; q < kSeTq; q++) {
                const uint4 x = *reinterpret_cast<const uint4 *>(&sm.sig[q][0]);
                const uint4 y = *reinterpret_cast<const uint4 *>(&sm.sig[q][4]);
                int l1 = __vsadu4(w[0], x.x);
                l1 += __vsadu4(w[1], x.y);
                l1 += __vsadu4(w[2], x.z);
                l1 += __vsadu4(w[3], x.w);
                l1 += __vsadu4(w[4], y.x);
                l1 += __vsadu4(w[5], y.y);
                l1 += __vsadu4(w[6], y.z);
                l1 += __vsadu4(w[7], y.w);
                const int R = sm.R[q];
                // ceil(l1 / 2) and the length difference bound the distance from below
                if (l1 <= 2 * R && abs(len - sm.qlen[q]) <= R) pass |= 1u << q;
            }
            if (tid >= n) pass = 0;
            // list the pairs: a scan over the CTA gives every thread its place
            const int c = __popc(pass);
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int z = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += z;
            }
            if (lane == 31) sm.wsum[warp] = incl;
            __syncthreads();
            int at = incl - c, total = 0;
#pragma unroll
            for (int v = 0; v < kSeThreads / 32; v++) {
                const int x = sm.wsum[v];
                if (v < warp) at += x;
                total += x;
            }
            for (uint32_t m = pass; m; m &= m - 1) sm.list[at++] = (unsigned short)((__ffs(m) - 1) << 8 | tid);
            __syncthreads();
            if (tid == 0) {
                tested += (unsigned long long)n * max(0, min(kSeTq, s.nq - q0));
                exact += (unsigned long long)total;
            }
            for (int i = tid; i < total; i += kSeThreads) {
                const int pr = sm.list[i], q = pr >> 8, r = pr & 255, R = sm.R[q];
                const int d = edit_words(sm.peq[q], sm.qlen[q], sm.text + r * kSeTextLd,
                                     t.tstrs + (size_t)sm.pos[r] * kStrStride, sm.len[r], R);
                if (d > R) continue;
                if (mode == kModeKnn) {
                    atomicAdd(&e.hist[(size_t)(q0 + q) * kSeHist + d], 1);
                    const int k = atomicAdd(&s.ccnt[q0 + q], 1);
                    if (k < s.cap) {
                        s.cpos[(size_t)(q0 + q) * s.cap + k] = sm.pos[r];
                        s.cv[(size_t)(q0 + q) * s.cap + k] = (float)d;
                    }
                } else if (mode == kModeRangeCount) {
                    atomicAdd(&sm.cnt[q], 1);
                } else {
                    const int id = t.id_list[sm.pos[r]], tq = s.a.qtime[s.bq[q0 + q]];
                    int wt = 0, wc = 0;
                    for (int j = s.a.ent_off[id], j1 = s.a.ent_off[id + 1]; j < j1; j++) {
                        const int4 v = s.a.ents[j];
                        wt += (v.x < tq && tq < v.y) ? 1 : 0;
                        wc += (v.z < tq && tq < v.w) ? 1 : 0;
                    }
                    if (wt) atomicAdd(&sm.cnt[q], wt);
                    if (wc) atomicAdd(&sm.cnt2[q], wc);
                }
            }
        }
        if (mode != kModeKnn) {
            __syncthreads();
            if (tid < kSeTq) {
                if (sm.cnt[tid]) atomicAdd(&s.cnt[q0 + tid], sm.cnt[tid]);
                if (sm.cnt2[tid]) atomicAdd(&s.cnt2[q0 + tid], sm.cnt2[tid]);
                sm.cnt[tid] = sm.cnt2[tid] = 0;
            }
        }
    }
    if (tid == 0 && s.a.stats && tested) {
        atomicAdd(&s.a.stats[0], tested);
        atomicAdd(&s.a.stats[2], exact);
    }
}

// ---------------------------------------------------------------- answers

__global__ void k_se_counts(EditArgs e)
{
    const SweepArgs &s = e.s;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s.nq) return;
    const int q = s.bq[i];
    if (e.qlen[i] >= 0) {
        s.a.counts[q] = s.cnt[i];
        if (s.a.mode == kModeRangeTimed) s.a.counts2[q] = s.cnt2[i];
        if (s.a.stats) atomicAdd(&s.a.stats[3], 1ull);
    }
}

// kNN answers of one sorted query per CTA: the listed objects up to the k-th
// distance (known exactly from the histogram), by (distance, id).
__global__ void __launch_bounds__(128) k_se_knn(EditArgs e)
{
    __shared__ unsigned long long key[kSeCap];
    __shared__ int s_n, s_R;
    const SweepArgs &s = e.s;
    const DevTree &t = s.a.t;
    const int i = blockIdx.x, tid = threadIdx.x, k = s.a.k;
    if (e.qlen[i] < 0) return;
    const int q = s.bq[i], m = s.ccnt[i];
    if (tid == 0) {
        const int *h = e.hist + (size_t)i * kSeHist;
        int R = kSeHist - 1, run = 0;
        for (int d = 0; d < kSeHist; d++) {
            run += h[d];
            if (run >= k) {
                R = d;
                break;
            }
        }
        s_R = R;
        s_n = 0;
    }
    __syncthreads();
    const int R = s_R;
    if (m > s.cap) {
        if (tid == 0) {
            const int at = atomicAdd(&s.ctr[1], 1);
            atomicAdd(&s.ctr[2], 1);
            s.left[at] = make_int4(q, 0, 0, 0);
            s.left_R[at] = (float)R;   // the exact k-th distance: another pass starts from it
        }
        return;
    }
    for (int c = tid; c < m; c += 128) {
        const int d = (int)s.cv[(size_t)i * s.cap + c];
        if (d <= R)
            key[atomicAdd(&s_n, 1)] = ((unsigned long long)(unsigned)d << 32) |
                                      (unsigned)t.id_list[s.cpos[(size_t)i * s.cap + c]];
    }
    __syncthreads();
    const int n = s_n;
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    for (int c = n + tid; c < p2; c += 128) key[c] = ~0ull;
    __syncthreads();
    for (int size = 2; size <= p2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int c = tid; c < p2 / 2; c += 128) {
                const int lo = 2 * c - (c & (stride - 1)), hi = lo + stride;
                const unsigned long long x = key[lo], y = key[hi];
                if ((x > y) == ((lo & size) == 0)) {
                    key[lo] = y;
                    key[hi] = x;
                }
            }
            __syncthreads();
        }
    for (int j = tid; j < k; j += 128) {
        const bool have = j < n;
        if (s.a.ids) s.a.ids[(size_t)q * k + j] = have ? (int)(uint32_t)key[j] : -1;
        if (s.a.dists) s.a.dists[(size_t)q * k + j] = have ? (float)(key[j] >> 32) : (float)t.infi_dis;
    }
    if (tid == 0) {
        s.a.kth[q] = n >= k ? (float)(key[k - 1] >> 32) : (float)t.infi_dis;
        if (s.a.stats) atomicAdd(&s.a.stats[3], 1ull);
    }
}

size_t plan_edit(const gts_index *idx, int tiles, int qnum, bool knn, unsigned char *base, EditArgs *out, void **cub,
                 size_t *cub_bytes)
{
    const int Qp = (tiles * kSeTq + 127) / 128 * 128;
    size_t off = 0, tb = 0;
    auto take = [&](size_t b) { size_t o = off; off += (b + 255) & ~(size_t)255; return base + o; };
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (int *)nullptr, (int *)nullptr, (int *)nullptr, (int *)nullptr, qnum, 0,
                                    32, (cudaStream_t)0);
    EditArgs e{};
    SweepArgs &r = e.s;
    r.Qp = Qp;
    r.tq = kSeTq;
    r.sample = 1;
    r.cap = kSeCap;
    r.left = (int4 *)take(sizeof(int4) * 2 * (size_t)qnum);
    r.left_R = (float *)take(4 * 2 * (size_t)qnum);
    r.ctr = (int *)take(64);
    r.nrows = (int *)take(4 * (size_t)tiles);
    r.key = (int *)take(4 * (size_t)qnum * 4);   // key, sorted key, identity, order: of the whole batch
    r.order = r.key + 3 * (size_t)qnum;
    r.bq = (int *)take(4 * (size_t)Qp);
    r.seed = (float *)take(4 * (size_t)qnum);
    r.R = (float *)take(4 * (size_t)Qp);
    r.ccnt = (int *)take(4 * (size_t)Qp * 3);
    r.cnt = r.ccnt + Qp;
    r.cnt2 = r.cnt + Qp;
    e.qlen = (int *)take(4 * (size_t)Qp);
    e.qpack = (uint32_t *)take(64 * (size_t)Qp);
    e.lens_ok = (uint4 *)take(sizeof(uint4) * (size_t)(Qp / kSeTq));
    r.lens_ok = e.lens_ok;
    e.qsig = (uint32_t *)take(32 * (size_t)Qp);
    r.dlo = (float *)take(4 * (size_t)std::max(idx->ncut_anc, 1) * Qp);
    r.dhi = (float *)take(4 * (size_t)std::max(idx->ncut_anc, 1) * Qp);
    r.rowpos = (int *)take(4 * (size_t)tiles * idx->num);
    if (knn) {
        e.hist = (int *)take(4 * (size_t)Qp * kSeHist);
        r.cpos = (int *)take(4 * (size_t)Qp * kSeCap);
        r.cv = (float *)take(4 * (size_t)Qp * kSeCap);
    }
    *cub = take(tb);
    *cub_bytes = tb;
    if (out) *out = e;
    return off;
}

template <typename W>
int edit_pass_words(gts_index *idx, EditArgs &e, cudaStream_t st)
{
    SweepArgs &s = e.s;
    int dev = 0, nsm = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    GTS_CUDA_TRY(cudaFuncSetAttribute(k_se_tile<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EditSmem<W>)));
    GTS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_se_tile<W>, kSeThreads, sizeof(EditSmem<W>)));
    s.ntiles = (s.nq + kSeTq - 1) / kSeTq;
    k_se_query<<<(s.Qp + 127) / 128, 128, 0, st>>>(e);
    if (s.nanc > 0) {
        // a CTA per query leaves the chip idle for few of them: split the pivots
        const int split = std::max(1, std::min((s.nanc + kSeThreads - 1) / kSeThreads, 2 * nsm / s.nq));
        k_se_pivots<W><<<dim3(s.nq, split), kSeThreads, 0, st>>>(e);
    }
    sweep_cut_launch(s, s.ntiles, st);
    k_se_tile<W><<<nsm * std::max(per_sm, 1), kSeThreads, sizeof(EditSmem<W>), st>>>(e);
    if (s.a.mode == kModeKnn) k_se_knn<<<s.nq, 128, 0, st>>>(e);
    else k_se_counts<<<(s.nq + 127) / 128, 128, 0, st>>>(e);
    idx->kernel_launches += 4 + (s.nanc > 0);
    GTS_CUDA_TRY(cudaGetLastError());
    return GTS_OK;
}

int edit_pass(gts_index *idx, EditArgs &e, cudaStream_t st)
{
    return e.wide ? edit_pass_words<unsigned long long>(idx, e, st) : edit_pass_words<uint32_t>(idx, e, st);
}

}  // namespace

// The sizes from which on the sweep is the sooner one.  Its launches take some
// 130 us for a tile and 220 for several, which a CTA of the traversal spends
// on 16,000 to 64,000 words, the fewer the smaller their leaves; only large
// batches of less pay.  Traversal and sweep, us, radius 2 where not given:
//   8,000 words, 1,000 queries  178  277    32,768, leaves of 3,300, 100 queries  174  217
//   16,384, 100 queries  138  204           32,768, small leaves, 100 queries     832  210
//   32,768, 8 queries    155  137           100,000, leaves of 10,000, 100 queries  441  207
// Radii far below the strings' lengths reach a leaf or two of a deep tree: words
// at radius 0, 200,000 of them, 1,000 queries: 204 and 294; strings of 20 to 50
// characters at radius 1, 60,000 of them, 100 queries: 114 and 307.  Strings of
// more than 64 characters are left to the traversal anyway.
static bool edit_sweep_pays(const gts_index *idx, const SearchArgs &a)
{
    const long long n = idx->num, q = a.qnum;
    const bool deep = n <= 32ll * idx->nleaf;
    if (2 * idx->str_lens[2] > n) return false;
    if (a.mode != kModeKnn && deep && floorf(std::min(a.r, 1e6f)) * 16.f * (float)n < (float)idx->str_lens[0]) return false;
    if (n * q >= 1 << 24) return true;
    return n >= (q <= kSeTq ? (deep ? 1 << 14 : 1 << 15) : (deep ? 1 << 15 : 1 << 16));
}

int run_sweep_edit(gts_index *idx, const SearchArgs &a, cudaStream_t st, int *done, const int4 **items, int *n_left)
{
    *done = 0;
    *n_left = 0;
    const int slot = a.mode == kModeRangeTimed ? kModeRangeCount : a.mode;
    const bool knn = a.mode == kModeKnn;
    if (a.deleted || a.items_in || a.seed_r2_bits || idx->ncut < 1 || idx->plain_pinned[slot] ||
        (!knn && idx->plain_split_set) || (knn ? a.k > 128 : !(a.r >= 0.f)) || !edit_sweep_pays(idx, a))
        return GTS_OK;
    const size_t budget = search_budget(idx);
    void *cub = nullptr;
    size_t cub_bytes = 0, bytes;
    int tiles = std::min(kSeMaxTiles, (a.qnum + kSeTq - 1) / kSeTq);
    for (;;) {
        bytes = plan_edit(idx, tiles, a.qnum, knn, nullptr, nullptr, &cub, &cub_bytes);
        if (bytes <= budget || tiles == 1) break;
        tiles = (tiles + 1) / 2;
    }
    if (bytes > budget || ensure_scratch(idx, bytes) != GTS_OK) return GTS_OK;
    EditArgs e;
    plan_edit(idx, tiles, a.qnum, knn, (unsigned char *)idx->scratch, &e, &cub, &cub_bytes);
    SweepArgs &s = e.s;
    e.tpack = idx->tpack;
    s.a = a;
    s.cut = idx->cut_node;
    s.ncut = idx->ncut;
    s.anc = idx->cut_anc;
    s.nanc = idx->ncut_anc;
    s.anc_idx = idx->cut_anc_idx;
    int pos_bits = 1, rc;
    while (pos_bits < 31 && (1 << pos_bits) < idx->num) pos_bits++;
    const int run = tiles * kSeTq;
    e.wide = 8 * idx->str_lens[1] > idx->num;   // many strings of more than 32 characters: one pass for all up to 64
    GTS_CUDA_TRY(cudaMemsetAsync(s.ctr, 0, 64, st));
    int *skey = s.key + a.qnum, *iota = skey + a.qnum;
    k_se_seed<<<a.qnum, kSeThreads, 0, st>>>(e, pos_bits);
    k_se_iota<<<(a.qnum + 255) / 256, 256, 0, st>>>(a.qnum, a.qnum > kSeTq ? iota : s.order);
    idx->kernel_launches += 2;
    if (a.qnum > kSeTq)
        GTS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(cub, cub_bytes, s.key, skey, iota, s.order, a.qnum, 0, 31, st));
    for (int q0 = 0; q0 < a.qnum; q0 += run) {
        s.q0 = q0;
        s.nq = std::min(run, a.qnum - q0);
        if ((rc = edit_pass(idx, e, st))) return rc;
    }
    auto outcome = [&](int *left, int *full, bool *ok) {
        int h[3] = {0, 0, 0}, status = 0;
        GTS_CUDA_TRY(cudaMemcpyAsync(h, s.ctr, sizeof(h), cudaMemcpyDeviceToHost, st));
        GTS_CUDA_TRY(cudaMemcpyAsync(&status, idx->d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
        GTS_CUDA_TRY(cudaStreamSynchronize(st));
        *left = h[1];
        *full = h[2];
        *ok = status == 0;
        return GTS_OK;
    };
    bool ok = false;
    int full = 0;   // queries left because their list was
    if ((rc = outcome(n_left, &full, &ok))) return rc;
    // once more: queries of 33 to 64 characters, and kNN queries whose lists
    // filled before their bound settled, from the exact k-th distance
    int4 *const lists[2] = {s.left, s.left + a.qnum};
    float *const bounds[2] = {s.left_R, s.left_R + a.qnum};
    for (int round = 0; round < kSeRounds && ok && (e.wide ? full : *n_left) > 0; round++) {
        const int n = *n_left;
        e.wide = 1;
        s.again = lists[round & 1];
        s.again_R = bounds[round & 1];
        s.left = lists[(round + 1) & 1];
        s.left_R = bounds[(round + 1) & 1];
        GTS_CUDA_TRY(cudaMemsetAsync(s.ctr, 0, 64, st));
        for (int q0 = 0; q0 < n; q0 += run) {
            s.q0 = q0;
            s.nq = std::min(run, n - q0);
            if ((rc = edit_pass(idx, e, st))) return rc;
        }
        if ((rc = outcome(n_left, &full, &ok))) return rc;
    }
    if (!ok) {   // a query id out of range: the traversal reports it
        GTS_CUDA_TRY(cudaMemsetAsync(idx->d_status, 0, sizeof(int), st));
        return GTS_OK;
    }
    *done = 1;
    *items = s.left;
    return GTS_OK;
}

}  // namespace gts
