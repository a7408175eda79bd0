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

}  // namespace

int seed_table_build(const FastSummary &bs, int nb, const FastShape &fs, cudaStream_t st)
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
    GTS_CUDA_TRY(cudaGetLastError());
    return GTS_OK;
}

}  // namespace gts
