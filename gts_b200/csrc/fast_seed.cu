// fast_seed.cu -- the seed table of the tensor-core kNN filter.
//
// Queries are objects, so a bound on a query's k-th distance can be computed
// per object ahead of any call: the k-th smallest distance from the object to
// the objects of its own block and of the kSeedNbr blocks whose centres lie
// nearest to its block's (the object itself counts, at distance 0).  Any k of
// those objects bound the query's k-th distance, and 32 blocks (4,096 objects)
// hold nearly all of a query's close neighbours, so the seed sits next to the
// answer: at 1,000,000 x 128 and k = 8 the filter lists 9.1 candidates per
// query against 97 from the own-block k-th distance.  Stored for k = 1, 2, 4,
// .., 64 (a call with another k reads the next power of two: a bound for the
// larger k bounds every smaller k).
//
// Both passes are all-pairs FP32 squared distances between 128 rows and
// 128-row tiles, so both run the same register tile: 256 threads, each 8 x 8
// pairs, rows staged 16 dimensions at a time by cp.async (two stages, row
// stride 20 floats: the quarter-warps' 16-byte reads fall into distinct
// banks).  A pair costs one subtraction and one fused multiply-add per
// dimension against 1/16 of a shared-memory read, so the FP32 pipe bounds
// them.  The distances are summed in dimension order (the reference's leaf
// loop order).
#include <algorithm>
#include <cfloat>
#include <climits>
#include "fast.cuh"

namespace gts {

namespace {

constexpr int kSdThreads = 256;
constexpr int kSdK = 16;               // dimensions per stage
constexpr int kSdLd = kSdK + 4;        // row stride in shared memory
constexpr int kSdPend = 64;            // values of one row waiting to be merged
constexpr int kSdMergeAt = 32;         // merge a row's waiting values from this many on
constexpr int kNbrKeep = 32;           // nearest centres kept per block (kSeedNbr of them used)
constexpr int kNbrPend = 64;
// Weak seeds: k = 2^kWkFirst on, more than 1.5 times (squared) the smallest of
// the neighbourhood; at most one object in kWkShare, and kWkMax in all, is
// looked at again, over its kWkBlocks nearest blocks.  Each reads every centre:
// kWkMax of them cost a few per cent of the seed table at any size.
constexpr int kWkFirst = 3, kWkCols = kSelfKN - kWkFirst;
constexpr float kWkRatio = 2.25f;
constexpr int kWkShare = 64, kWkMax = 4096;
constexpr int kWkBlocks = 8;

static_assert(kSeedBest == 64 && kSdPend == 64 && kSeedNbr <= kNbrKeep, "list sizes");

struct SeedTiles {
    float a[2][kFB * kSdLd], b[2][kFB * kSdLd];
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// 128 rows (those past n repeat row n - 1) x 16 dimensions from k0.
__device__ __forceinline__ void stage_rows(float *dst, const float *rows, int n, int kp, int k0)
{
#pragma unroll
    for (int u = 0; u < kFB * 4 / kSdThreads; u++) {
        const int i = threadIdx.x + u * kSdThreads, r = i >> 2, j = i & 3;
        cp_async16(dst + r * kSdLd + 4 * j, rows + (size_t)min(r, n - 1) * kp + k0 + 4 * j);
    }
}

// acc[i][c] += squared differences of rows a[tq + 16 i] and b[to + 16 c] over
// the staged dimensions.
__device__ __forceinline__ void tile_add(const float *a, const float *b, int tq, int to, float (&acc)[8][8])
{
#pragma unroll 2   // fully unrolled the loop misses the instruction cache: 54.4 ms of seeds instead of 51.0
    for (int k = 0; k < kSdK; k += 4) {
        float4 o[8];
#pragma unroll
        for (int c = 0; c < 8; c++) o[c] = *reinterpret_cast<const float4 *>(b + (to + 16 * c) * kSdLd + k);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float4 q = *reinterpret_cast<const float4 *>(a + (tq + 16 * i) * kSdLd + k);
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float e0 = o[c].x - q.x, e1 = o[c].y - q.y, e2 = o[c].z - q.z, e3 = o[c].w - q.w;
                acc[i][c] = fmaf(e3, e3, fmaf(e2, e2, fmaf(e1, e1, fmaf(e0, e0, acc[i][c]))));
            }
        }
    }
}

// One compare-exchange of a bitonic network across the warp's lanes.
template <typename T>
__device__ __forceinline__ T exchange(T v, int stride, bool up, int lane)
{
    const T o = __shfl_xor_sync(0xffffffffu, v, stride);
    const bool low = (lane & stride) == 0;
    return (low == up) ? (o < v ? o : v) : (o < v ? v : o);
}

// Sorts 64 values, element r * 32 + lane in v[r], descending.
template <typename T>
__device__ __forceinline__ void sort64_desc(T (&v)[2], int lane)
{
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            v[0] = exchange(v[0], stride, size == 32 ? false : (lane & size) != 0, lane);
            v[1] = exchange(v[1], stride, size == 32 ? true : (lane & size) != 0, lane);
        }
    const T lo = v[1] < v[0] ? v[1] : v[0], hi = v[1] < v[0] ? v[0] : v[1];
    v[0] = hi;
    v[1] = lo;
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
        v[0] = exchange(v[0], stride, false, lane);
        v[1] = exchange(v[1], stride, false, lane);
    }
}

// The 64 smallest of best (ascending, 64 values) and n <= 64 others, ascending.
template <typename T>
__device__ __forceinline__ void merge64(T *best, const T *pend, int n, T none, int lane)
{
    T p[2] = {lane < n ? pend[lane] : none, lane + 32 < n ? pend[lane + 32] : none};
    sort64_desc(p, lane);
    T v[2] = {best[lane], best[lane + 32]};
    v[0] = p[0] < v[0] ? p[0] : v[0];   // ascending against descending: the smaller half, bitonic
    v[1] = p[1] < v[1] ? p[1] : v[1];
    const T lo = v[1] < v[0] ? v[1] : v[0], hi = v[1] < v[0] ? v[0] : v[1];
    v[0] = lo;
    v[1] = hi;
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
        v[0] = exchange(v[0], stride, true, lane);
        v[1] = exchange(v[1], stride, true, lane);
    }
    best[lane] = v[0];
    best[lane + 32] = v[1];
}

struct SelfkSmem {
    SeedTiles t;
    float best[kFB][kSeedBest];   // per object, ascending
    float pend[kFB][kSdPend];
    int pcnt[kFB];
    unsigned omask[kFB / 32], vmask[2][kFB / 32];
};

// The seed table: one CTA per block b, over b itself and its neighbours.  A
// value below the object's 64th smallest so far waits in pend; a warp merges a
// row's waiting values (a 64-value bitonic sort and merge) when 32 have come
// or a value found no room, and the values without room try again.
// Two CTAs fit an SM, so one merges while the other multiplies.  At
// 1,000,000 x 128: 51 ms, of which the FP32 pipe needs 31 and the merges 5
// (165 ms with a warp per object, 4 pairs per lane, a rank-by-counting merge
// at every block).
__global__ void __launch_bounds__(kSdThreads, 2) k_fast_selfk(FastSummary bs, int kp, const int *__restrict__ nbr)
{
    extern __shared__ __align__(16) unsigned char sd_smem[];
    SelfkSmem &s = *reinterpret_cast<SelfkSmem *>(sd_smem);
    const int b = blockIdx.x, t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int tq = t & 15, to = t >> 4;
    const float *arow = bs.prow + (size_t)b * kFB * kp;
    const int nc = kp / kSdK;
    if (t < kFB) {
        const unsigned m = __ballot_sync(0xffffffffu, bs.ids[b * kFB + t] >= 0);
        if (lane == 0) s.omask[warp] = m;
        s.pcnt[t] = 0;
    }
    for (int i = t; i < kFB * kSeedBest; i += kSdThreads) (&s.best[0][0])[i] = FLT_MAX;
    int nlist = 1;   // the blocks in use: b, then its neighbours (packed at the front)
    while (nlist <= kSeedNbr && nbr[(size_t)b * kSeedNbr + nlist - 1] >= 0) nlist++;
    auto block_at = [&](int i) { return i == 0 ? b : nbr[(size_t)b * kSeedNbr + i - 1]; };
    auto issue = [&](int step) {
        const int i = step / nc, k0 = (step - i * nc) * kSdK;
        stage_rows(s.t.a[step & 1], arow, kFB, kp, k0);
        stage_rows(s.t.b[step & 1], bs.prow + (size_t)block_at(i) * kFB * kp, kFB, kp, k0);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int cnt = 0, step = 0;   // cnt: objects in the blocks used so far
    const int steps = nlist * nc;
    issue(0);
    for (int i = 0; i < nlist; i++) {
        const int j = block_at(i);
        if (t < kFB) {
            const unsigned m = __ballot_sync(0xffffffffu, bs.ids[j * kFB + t] >= 0);
            if (lane == 0) s.vmask[i & 1][warp] = m;
        }
        float acc[8][8];
#pragma unroll
        for (int q = 0; q < 8; q++)
#pragma unroll
            for (int c = 0; c < 8; c++) acc[q][c] = 0.f;
        for (int ch = 0; ch < nc; ch++, step++) {
            // the stage has come, and everyone is done with the other one
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (step + 1 < steps) issue(step + 1);
            tile_add(s.t.a[step & 1], s.t.b[step & 1], tq, to, acc);
        }
        // values that may rank: valid rows, below the row's 64th so far
        unsigned valid = 0;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int o = to + 16 * c;
            valid |= ((s.vmask[i & 1][o >> 5] >> (o & 31)) & 1u) << c;
        }
#pragma unroll
        for (int w = 0; w < kFB / 32; w++) cnt += __popc(s.vmask[i & 1][w]);
        unsigned long long todo = 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int row = tq + 16 * q;
            if ((s.omask[row >> 5] >> (row & 31)) & 1u) todo |= (unsigned long long)valid << (8 * q);
        }
        for (;;) {
            bool full = false;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int row = tq + 16 * q;
                const float thr = s.best[row][kSeedBest - 1];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    if (!((todo >> (8 * q + c)) & 1ull)) continue;
                    bool done = true;
                    if (acc[q][c] < thr) {
                        const int at = atomicAdd(&s.pcnt[row], 1);
                        if (at < kSdPend) s.pend[row][at] = acc[q][c];
                        else done = false;
                    }
                    if (done) todo &= ~(1ull << (8 * q + c));
                    else full = true;
                }
            }
            const int any = __syncthreads_or(full);
            for (int row = warp; row < kFB; row += kSdThreads / 32) {
                const int n = s.pcnt[row];
                if (n < kSdMergeAt && i + 1 < nlist) continue;
                if (n > 0) {
                    merge64(s.best[row], s.pend[row], min(n, kSdPend), FLT_MAX, lane);
                    __syncwarp();
                    if (lane == 0) s.pcnt[row] = 0;
                }
            }
            __syncthreads();
            if (!any) break;
        }
    }
    // A sum of at most 320 non-negative FP32 terms is within 322 * 2^-24 <
    // 2e-5 relative of the exact sum of the same FP32 differences squared, the
    // value the reference's FP64 sum rounds, so widening by (1 + 4e-5) gives a
    // certified bound on the reference's k-th squared distance.  FLT_MAX where
    // the blocks hold fewer than k objects (no seed).
    for (int e = t; e < kFB * kSelfK; e += kSdThreads) {
        const int m = e / kSelfK, jk = e % kSelfK;
        int v = __float_as_int(FLT_MAX);
        if (jk < kSelfKN && ((s.omask[m >> 5] >> (m & 31)) & 1u) && cnt >= (1 << jk))
            v = __float_as_int(s.best[m][(1 << jk) - 1] * (1.f + 4e-5f));
        bs.selfk[((size_t)b * kFB + m) * kSelfK + jk] = v;
    }
}

struct NbrSmem {
    SeedTiles t;
    unsigned long long best[kFB][2 * kNbrKeep];   // (distance bits, block), ascending; 64 wide for the merge
    unsigned long long pend[kFB][kNbrPend];
    int pcnt[kFB];
};

// The nearest centres of 128 blocks among slice y of the centre tiles: the 64
// smallest (squared distance, block id) keys, of which the first kNbrKeep go
// to part[y][block].  Ties go to the smaller block id.
__global__ void __launch_bounds__(kSdThreads, 1) k_fast_nbrs(FastSummary bs, int nb, int kp,
                                                             unsigned long long *__restrict__ part)
{
    extern __shared__ __align__(16) unsigned char sd_smem[];
    NbrSmem &s = *reinterpret_cast<NbrSmem *>(sd_smem);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, tq = t & 15, to = t >> 4;
    const int b0 = blockIdx.x * kFB, nt = (nb + kFB - 1) / kFB, nc = kp / kSdK;
    const int t0 = (int)((long long)nt * blockIdx.y / gridDim.y), t1 = (int)((long long)nt * (blockIdx.y + 1) / gridDim.y);
    const unsigned long long none = ~0ull;
    for (int i = t; i < kFB * 2 * kNbrKeep; i += kSdThreads) (&s.best[0][0])[i] = none;
    if (t < kFB) s.pcnt[t] = 0;
    __syncthreads();
    auto issue = [&](int step) {
        const int i = t0 + step / nc, k0 = (step % nc) * kSdK;
        stage_rows(s.t.a[step & 1], bs.cen + (size_t)b0 * kp, nb - b0, kp, k0);
        stage_rows(s.t.b[step & 1], bs.cen + (size_t)i * kFB * kp, nb - i * kFB, kp, k0);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int step = 0;
    const int steps = (t1 - t0) * nc;
    if (steps > 0) issue(0);
    for (int i = t0; i < t1; i++) {
        float acc[8][8];
#pragma unroll
        for (int q = 0; q < 8; q++)
#pragma unroll
            for (int c = 0; c < 8; c++) acc[q][c] = 0.f;
        for (int ch = 0; ch < nc; ch++, step++) {
            // the stage has come, and everyone is done with the other one
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (step + 1 < steps) issue(step + 1);
            tile_add(s.t.a[step & 1], s.t.b[step & 1], tq, to, acc);
        }
        unsigned long long todo = 0;
#pragma unroll
        for (int q = 0; q < 8; q++)
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const int j = i * kFB + to + 16 * c, b = b0 + tq + 16 * q;
                if (j < nb && b < nb && j != b && acc[q][c] < FLT_MAX) todo |= 1ull << (8 * q + c);
            }
        for (;;) {
            bool full = false;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int row = tq + 16 * q;
                const unsigned long long thr = s.best[row][kNbrKeep - 1];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    if (!((todo >> (8 * q + c)) & 1ull)) continue;
                    const unsigned long long key =
                        ((unsigned long long)__float_as_uint(acc[q][c]) << 32) | (unsigned)(i * kFB + to + 16 * c);
                    bool done = true;
                    if (key < thr) {
                        const int at = atomicAdd(&s.pcnt[row], 1);
                        if (at < kNbrPend) s.pend[row][at] = key;
                        else done = false;
                    }
                    if (done) todo &= ~(1ull << (8 * q + c));
                    else full = true;
                }
            }
            const int any = __syncthreads_or(full);
            for (int row = warp; row < kFB; row += kSdThreads / 32) {
                const int n = s.pcnt[row];
                if (n < kSdMergeAt && i + 1 < t1) continue;
                if (n > 0) {
                    merge64(s.best[row], s.pend[row], min(n, kNbrPend), none, lane);
                    __syncwarp();
                    if (lane == 0) s.pcnt[row] = 0;
                }
            }
            __syncthreads();
            if (!any) break;
        }
    }
    for (int e = t; e < kFB * kNbrKeep; e += kSdThreads) {
        const int b = b0 + e / kNbrKeep;
        if (b < nb) part[((size_t)blockIdx.y * nb + b) * kNbrKeep + e % kNbrKeep] = s.best[e / kNbrKeep][e % kNbrKeep];
    }
}

// One warp per block: the kSeedNbr nearest centres of all slices (-1: none).
__global__ void __launch_bounds__(256) k_fast_nbrs_merge(int nb, int slices, const unsigned long long *__restrict__ part,
                                                         int *__restrict__ nbr)
{
    __shared__ unsigned long long lists[8][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.x * 8 + warp;
    if (b >= nb) return;
    unsigned long long *best = lists[warp];
    best[lane] = best[lane + 32] = ~0ull;
    __syncwarp();
    for (int y = 0; y < slices; y++) {
        merge64(best, part + ((size_t)y * nb + b) * kNbrKeep, kNbrKeep, ~0ull, lane);
        __syncwarp();
    }
    if (lane < kSeedNbr) nbr[(size_t)b * kSeedNbr + lane] = best[lane] == ~0ull ? -1 : (int)(uint32_t)best[lane];
}

// Smallest seed of each block for k = 8 .. 64 (float bits).
__global__ void __launch_bounds__(kFB) k_fast_seed_min(FastSummary bs, int *__restrict__ bmin)
{
    __shared__ int part[kFB / 32][kWkCols];
    const int b = blockIdx.x, t = threadIdx.x, slot = b * kFB + t;
    const bool live = bs.ids[slot] >= 0;
#pragma unroll
    for (int c = 0; c < kWkCols; c++) {
        const int v = __reduce_min_sync(0xffffffffu, live ? bs.selfk[(size_t)slot * kSelfK + kWkFirst + c] : INT_MAX);
        if ((t & 31) == 0) part[t >> 5][c] = v;
    }
    __syncthreads();
    if (t < kWkCols) bmin[b * kWkCols + t] = min(min(part[0][t], part[1][t]), min(part[2][t], part[3][t]));
}

// Objects whose seed is far above the smallest of their block and its
// neighbours (cnt counts them, the first cap are listed by slot).
__global__ void __launch_bounds__(kFB) k_fast_weak_list(FastSummary bs, const int *__restrict__ bmin, int cap,
                                                        int *__restrict__ list, int *__restrict__ cnt)
{
    __shared__ float ref[kWkCols];
    const int b = blockIdx.x, t = threadIdx.x, lane = t & 31, slot = b * kFB + t;
    static_assert(kSeedNbr == 31 && kWkCols == kFB / 32, "a warp per column, a lane per block");
    const int j = lane < kSeedNbr ? bs.nbr[(size_t)b * kSeedNbr + lane] : b;
    const int m = __reduce_min_sync(0xffffffffu, j >= 0 ? bmin[j * kWkCols + (t >> 5)] : INT_MAX);
    if (lane == 0) ref[t >> 5] = __int_as_float(m);
    __syncthreads();
    if (bs.ids[slot] < 0) return;
    bool weak = false;
#pragma unroll
    for (int c = 0; c < kWkCols; c++)
        weak |= __int_as_float(bs.selfk[(size_t)slot * kSelfK + kWkFirst + c]) > kWkRatio * ref[c];
    if (!weak) return;
    const int at = atomicAdd(cnt, 1);
    if (at < cap) list[at] = slot;
}

// Squared distance of x (shared, kp floats) to the rows at p and the next
// three, ld apart, in every lane.
__device__ __forceinline__ void dist4(const float *x, const float *p, size_t ld, int n, int kp, int lane, float (&s)[4])
{
#pragma unroll
    for (int u = 0; u < 4; u++) s[u] = 0.f;
    for (int d = 4 * lane; d < kp; d += 128) {
        const float4 a = *reinterpret_cast<const float4 *>(x + d);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float4 o = *reinterpret_cast<const float4 *>(p + (size_t)min(u, n - 1) * ld + d);
            const float e0 = o.x - a.x, e1 = o.y - a.y, e2 = o.z - a.z, e3 = o.w - a.w;
            s[u] = fmaf(e3, e3, fmaf(e2, e2, fmaf(e1, e1, fmaf(e0, e0, s[u]))));
        }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], m);
}

// Better seeds for the listed objects, one CTA each: the k-th distances over
// the objects of the kWkBlocks blocks whose centres lie nearest to the object
// itself.  A block that halving left across two groups has its neighbours
// around its centre, so the few objects of the smaller group get seeds that
// reach over half of the data: 2 of 10,000 queries at 1,000,000 x 128 made
// 16,000 of the 33,500 (tile, block) entries of their filter run and 280 of
// its 780 us.  The centres are read once per listed object (4.4 MB there, from
// L2), which is why their number is bounded.
__global__ void __launch_bounds__(kSdThreads) k_fast_weak(FastSummary bs, int nb, int kp, int cap,
                                                          const int *__restrict__ list, const int *__restrict__ cnt)
{
    __shared__ __align__(16) float x[kFMaxKp];
    __shared__ __align__(16) float d[kWkBlocks * kFB];
    __shared__ unsigned long long key[8 * kWkBlocks];
    __shared__ int sel[kWkBlocks];
    static_assert(kSdThreads == 32 * 8 && kWkBlocks == 8, "a warp per chosen block");
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, n = min(*cnt, cap);
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const int slot = list[e];
        __syncthreads();
        for (int i = t; i < kp; i += kSdThreads) x[i] = bs.prow[(size_t)slot * kp + i];
        __syncthreads();
        // the warp's nearest centres, ascending over the lanes
        unsigned long long mine = ~0ull;
        for (int j0 = 4 * warp; j0 < nb; j0 += 32) {
            float s[4];
            dist4(x, bs.cen + (size_t)j0 * kp, kp, nb - j0, kp, lane, s);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const unsigned long long v = ((unsigned long long)__float_as_uint(s[u]) << 32) | (unsigned)(j0 + u);
                if (j0 + u >= nb || v >= __shfl_sync(0xffffffffu, mine, kWkBlocks - 1)) continue;
                const int at = __popc(__ballot_sync(0xffffffffu, mine < v));
                const unsigned long long up = __shfl_up_sync(0xffffffffu, mine, 1);
                if (lane >= at) mine = lane == at ? v : up;
            }
        }
        if (lane < kWkBlocks) key[warp * kWkBlocks + lane] = mine;
        if (t < kWkBlocks) sel[t] = -1;
        __syncthreads();
        if (t < 8 * kWkBlocks && key[t] != ~0ull) {
            int r = 0;
            for (int i = 0; i < 8 * kWkBlocks; i++) r += key[i] < key[t];
            if (r < kWkBlocks) sel[r] = (int)(uint32_t)key[t];
        }
        __syncthreads();
        const int b = sel[warp];
        for (int r = 0; r < kFB; r += 4) {
            float s[4] = {FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX};
            if (b >= 0) dist4(x, bs.prow + ((size_t)b * kFB + r) * kp, kp, 4, kp, lane, s);
            if (lane < 4)
                d[warp * kFB + r + lane] = b >= 0 && bs.ids[b * kFB + r + lane] >= 0
                                               ? (lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3])
                                               : FLT_MAX;
        }
        __syncthreads();
        // ranks, ties by position
        float v[4];
        int rk[4] = {0, 0, 0, 0};
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = d[t + u * kSdThreads];
        for (int i = 0; i < kWkBlocks * kFB; i += 4) {
            const float4 o = *reinterpret_cast<const float4 *>(d + i);
            const float oo[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int w = 0; w < 4; w++)
#pragma unroll
                for (int u = 0; u < 4; u++)
                    rk[u] += oo[w] < v[u] || (oo[w] == v[u] && i + w < t + u * kSdThreads);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = rk[u] + 1;
            if (k > kSeedBest || (k & (k - 1)) || !(v[u] < FLT_MAX)) continue;
            int *out = bs.selfk + (size_t)slot * kSelfK + (31 - __clz(k));
            *out = min(*out, __float_as_int(v[u] * (1.f + 4e-5f)));   // widened like every seed
        }
    }
}

}  // namespace

size_t seed_table_scratch(int nb, int num)
{
    return sizeof(int) * ((size_t)nb * kWkCols + 1 + num / kWkShare + 1);
}

int seed_table_build(const FastSummary &bs, int nb, int num, const FastShape &fs, int *scratch, cudaStream_t st)
{
    // slices of the centre tiles: enough CTAs for every SM; a slice writes
    // kNbrKeep keys per block into the seed table's own bytes (not made yet)
    constexpr int kSliceCap = (int)(sizeof(int) * kFB * kSelfK / (sizeof(unsigned long long) * kNbrKeep));
    const int nt = (nb + kFB - 1) / kFB;
    const int slices = std::max(1, std::min(std::min(kSliceCap, nt), (148 + nt - 1) / nt));
    unsigned long long *part = reinterpret_cast<unsigned long long *>(bs.selfk);
    GTS_CUDA_TRY(cudaFuncSetAttribute(k_fast_nbrs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(NbrSmem)));
    GTS_CUDA_TRY(cudaFuncSetAttribute(k_fast_selfk, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(SelfkSmem)));
    k_fast_nbrs<<<dim3(nt, slices), kSdThreads, sizeof(NbrSmem), st>>>(bs, nb, fs.kp, part);
    k_fast_nbrs_merge<<<(nb + 7) / 8, 256, 0, st>>>(nb, slices, part, bs.nbr);
    k_fast_selfk<<<nb, kSdThreads, sizeof(SelfkSmem), st>>>(bs, fs.kp, bs.nbr);
    int *bmin = scratch, *cnt = bmin + (size_t)nb * kWkCols, *list = cnt + 1;
    const int cap = std::min(num / kWkShare, kWkMax) + 1;
    GTS_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int), st));
    k_fast_seed_min<<<nb, kFB, 0, st>>>(bs, bmin);
    k_fast_weak_list<<<nb, kFB, 0, st>>>(bs, bmin, cap, list, cnt);
    k_fast_weak<<<std::min(cap, 148 * 8), kSdThreads, 0, st>>>(bs, nb, fs.kp, cap, list, cnt);
    GTS_CUDA_TRY(cudaGetLastError());
    return GTS_OK;
}

}  // namespace gts
