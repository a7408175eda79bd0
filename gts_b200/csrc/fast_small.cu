// fast_small.cu -- the fast form for a few queries.
//
// The tensor-core filter answers tiles of 128 queries; for one query its nine
// dependent kernels are 127 / 128 padding and took 200 us at 50,000 x 300 (231
// us for the host call), with one CTA in most of them.  The seed table and the
// block balls serve a few queries as well without tiles, in three launches
// over the whole chip:
//
//   * k_small_prune: a warp per block centre measures it against up to eight
//     queries at once and lists the blocks within reach of their seeds;
//   * k_small_rows: a warp per eight rows of the listed blocks, FP32 distances
//     against the seed with the sweep's bounds (sweep.cuh);
//   * k_small_final: a CTA per query, the reference's arithmetic on what is
//     left, as the sweep's last kernel.
//
// Queries the lists cannot hold go back to the caller.  The counters of a call
// are cleared by its last CTA, so a call needs no clearing launch.
#include <algorithm>
#include "fast.cuh"
#include "sweep.cuh"

namespace gts {

namespace {

constexpr int kSmGroup = 8;      // queries a warp measures a centre against

struct SmallArgs {
    DevTree t;
    FastSummary bs;
    int nb, kp;
    const int *qids;
    int qnum, k, jk;
    const int *carry;            // nullable: bounds reached before (squared, float bits)
    int *nblk, *ccnt;            // per query: listed blocks, candidates
    int *ticket, *nfail;
    int *blist;                  // [qnum][nb]
    int *cpos;                   // [qnum][kSwCap] slots
    float *cv;
    float *kth, *dists;
    int *ids, *fail;
    int *result;                 // [0] queries listed in fail (host memory)
    unsigned long long *stats;
    int reset;                   // the call's first pass: statistics start from zero
};

// Upper bound on the query's k-th distance from its seed; negative: bad id.
__device__ __forceinline__ float small_radius(const SmallArgs &a, int q)
{
    const int qid = a.qids[q];
    if (qid < 0 || qid >= a.t.num) return -1.f;
    int r2 = a.bs.selfk[(size_t)a.bs.pos[qid] * kSelfK + a.jk];
    if (a.carry) r2 = min(r2, a.carry[q]);   // non-negative floats order like their bits
    return sqrtf(__int_as_float(r2)) * (1.f + 1e-6f) + 1e-18f;
}

// Eight sums over the warp at once: lane l returns the sum of v[l >> 2].
__device__ __forceinline__ float warp_sum8(float (&v)[8], int lane)
{
#pragma unroll
    for (int w = 4; w >= 1; w >>= 1) {
        const int o = w * 4;   // 16, 8, 4
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < w; i++) {
            const float send = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}

template <int NX>
__global__ void __launch_bounds__(256) k_small_prune(SmallArgs a)
{
    __shared__ float qr[kSmGroup][NX * 32];
    __shared__ float R[kSmGroup];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q0 = blockIdx.y * kSmGroup;
    if (a.reset && blockIdx.x == 0 && blockIdx.y == 0 && tid < kStatsN) a.stats[tid] = 0;
    if (tid < kSmGroup) R[tid] = q0 + tid < a.qnum ? small_radius(a, q0 + tid) : -1.f;
    __syncthreads();
    for (int i = tid; i < kSmGroup * NX * 32; i += 256) {
        const int q = i / (NX * 32), j = i % (NX * 32);
        qr[q][j] = R[q] >= 0.f && j < a.t.dim ? a.t.rows[(size_t)a.qids[q0 + q] * a.t.dim + j] : 0.f;
    }
    __syncthreads();
    const float g = 2.f * f32_sum_rel_bound(a.kp + 32) + 4.f * 5.9604645e-8f;
    for (int b = blockIdx.x * 8 + warp; b < a.nb; b += gridDim.x * 8) {
        float c[NX];
#pragma unroll
        for (int i = 0; i < NX; i++) c[i] = lane + 32 * i < a.kp ? a.bs.cen[(size_t)b * a.kp + lane + 32 * i] : 0.f;
        const float rad = a.bs.rad[b];
        float v[kSmGroup];
#pragma unroll
        for (int q = 0; q < kSmGroup; q++) {
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < NX; i++) {
                const float d = c[i] - qr[q][lane + 32 * i];
                s = fmaf(d, d, s);
            }
            v[q] = s;
        }
        const float d2 = warp_sum8(v, lane);
        const int q = lane >> 2;
        if ((lane & 3) == 0 && rad >= 0.f && R[q] >= 0.f) {
            const float lo = sqrtf(fmaxf(d2 - kSwTiny, 0.f) * (1.f - g)) * (1.f - 4e-7f);
            if (!(lo > (rad + R[q]) * (1.f + 1e-6f)))
                a.blist[(size_t)(q0 + q) * a.nb + atomicAdd(&a.nblk[q0 + q], 1)] = b;
        }
    }
}

__global__ void __launch_bounds__(256) k_small_rows(SmallArgs a)
{
    extern __shared__ __align__(16) float sq[];   // the query row, zero padded to kp
    const int q = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = a.nblk[q];
    if ((int)blockIdx.x >= 2 * n) return;   // also: a bad id lists no block
    const int qid = a.qids[q];
    for (int j = tid; j < a.kp; j += 256) sq[j] = j < a.t.dim ? a.t.rows[(size_t)qid * a.t.dim + j] : 0.f;
    __syncthreads();
    const float R = small_radius(a, q);
    const double g = 2.0 * (double)f32_sum_rel_bound(a.kp + 32) + 4.0 * 5.9604645e-8;
    const double top = (double)R * R * (1.0 + 4e-6) / (1.0 - g) + 4.0 * kSwTiny;
    const float vthr = top < FLT_MAX ? __double2float_ru(top) : FLT_MAX;
    const int self = a.bs.pos[qid];
    // a half block (64 rows) per step: eight rows per warp
    for (int h = blockIdx.x; h < 2 * n; h += gridDim.x) {
        const int b = a.blist[(size_t)q * a.nb + (h >> 1)];
        const int s0 = b * kFB + (h & 1) * 64 + warp * 8;
        const float *rp[8];
#pragma unroll
        for (int u = 0; u < 8; u++) rp[u] = a.bs.prow + (size_t)(s0 + u) * a.kp;
        float v[8];
        warp_row_values<8>(rp, sq, a.kp, kL2, lane, v);
        float mine = 0.f;
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (lane == u) mine = v[u];
        if (lane < 8) {
            const int slot = s0 + lane;
            if (a.bs.ids[slot] >= 0 && (mine <= vthr || slot == self)) {
                const int at = atomicAdd(&a.ccnt[q], 1);
                if (at < kSwCap) {
                    a.cpos[(size_t)q * kSwCap + at] = slot;
                    a.cv[(size_t)q * kSwCap + at] = slot == self ? 0.f : mine;
                }
            }
        }
    }
}

__global__ void __launch_bounds__(128) k_small_final(SmallArgs a)
{
    extern __shared__ __align__(16) unsigned char sm_smem[];
    FinalSmem &f = *reinterpret_cast<FinalSmem *>(sm_smem);
    const int q = blockIdx.x, tid = threadIdx.x, k = a.k;
    const int m = a.ccnt[q], nblk = a.nblk[q];
    const int qid = a.qids[q];
    const bool ok = qid >= 0 && qid < a.t.num;
    const int self = ok ? a.bs.pos[qid] : -1;
    if (tid == 0) f.n = 0;
    __syncthreads();
    // a full list, or fewer than k objects within the seed: not answered here
    const bool failed = !ok || m > kSwCap || (m < k && m < a.t.num);
    int n = 0;
    if (!failed) {
        const int *cpos = a.cpos + (size_t)q * kSwCap;
        const float *cv = a.cv + (size_t)q * kSwCap;
        for (int c = tid; c < m; c += 128) f.key[c] = __float_as_uint(cpos[c] == self ? 0.f : sw_hi(kL2, a.kp, cv[c]));
        __syncthreads();
        float B = FLT_MAX;
        if (m > k) B = __uint_as_float(cta_kth(f.key, m, k, f.hist));
        for (int c = tid; c < m; c += 128)
            if (cpos[c] == self || sw_lo(kL2, a.kp, cv[c]) <= B) f.pos[atomicAdd(&f.n, 1)] = cpos[c];
        __syncthreads();
        n = f.n;
        const float *qrow = a.t.rows + (size_t)qid * a.t.dim;
        exact_knn(f, kL2, a.t.dim, a.bs.prow, (size_t)a.kp, a.bs.ids, self, qrow, n, k);
        for (int j = tid; j < k; j += 128) {
            const bool have = j < n;
            if (a.ids) a.ids[(size_t)q * k + j] = have ? f.id[j] : -1;
            if (a.dists) a.dists[(size_t)q * k + j] = have ? (float)f.d[j] : (float)a.t.infi_dis;
        }
        if (tid == 0) a.kth[q] = n >= k ? (float)f.d[k - 1] : (float)a.t.infi_dis;
    }
    if (tid == 0) {
        atomicAdd(&a.stats[0], (unsigned long long)nblk);
        atomicAdd(&a.stats[1], (unsigned long long)nblk * kFB * a.kp * 4);
        atomicAdd(&a.stats[2], (unsigned long long)n);
        atomicAdd(&a.stats[5], (unsigned long long)m);
        atomicAdd(&a.stats[7], (unsigned long long)a.nb);
        a.nblk[q] = 0;
        a.ccnt[q] = 0;
        if (failed) a.fail[atomicAdd(a.nfail, 1)] = q;
        __threadfence();
        if (atomicAdd(a.ticket, 1) == (int)gridDim.x - 1) {   // the last query
            __threadfence();
            a.result[0] = atomicAdd(a.nfail, 0);
            __threadfence_system();
            *a.nfail = 0;
            *a.ticket = 0;
            atomicAdd(&a.stats[6], 1ull);
        }
    }
}

}  // namespace

// The handle's buffers for small batches: device lists, and the result word
// in host memory.
size_t fast_small_bytes(const gts_index *idx)
{
    return 1024 + 4 * (size_t)kSmallMax * ((size_t)idx->fast_nb + 1 + 2 * kSwCap + 2);
}

static int small_buffers(gts_index *idx, cudaStream_t st)
{
    const size_t need = fast_small_bytes(idx);
    if (!idx->small_result && cudaHostAlloc((void **)&idx->small_result, 64, cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        idx->small_result = nullptr;
        gts_set_error("cudaHostAlloc of a result word failed");
        return GTS_ERR_NOMEM;
    }
    if (idx->small_bytes >= need) return GTS_OK;
    if (idx->small_buf) dev_free(idx->small_buf);
    idx->small_buf = nullptr;
    idx->small_bytes = 0;
    if (dev_malloc(&idx->small_buf, need) != cudaSuccess) {
        cudaGetLastError();
        idx->small_buf = nullptr;
        gts_set_error("cudaMalloc of %zu bytes for small batches failed", need);
        return GTS_ERR_NOMEM;
    }
    idx->small_bytes = need;
    GTS_CUDA_TRY(cudaMemsetAsync(idx->small_buf, 0, 1024, st));   // the counters
    return GTS_OK;
}

bool fast_small_takes(const gts_index *idx, int qnum)
{
    // each query reads its blocks' rows for itself: 64 queries of 128 dimensions
    // 0.6 of the tiles' time, of 300 325 us against 285 (33 of them 209 against 286)
    if (qnum * fast_shape(idx->dim).kp > 1 << 14) return false;
    // a group of eight queries reads every block centre: past about 2^17 of
    // those reads (64 MB at 128 dimensions) the tiles are as fast
    return qnum >= 1 && qnum <= kSmallMax && (long long)((qnum + kSmGroup - 1) / kSmGroup) * idx->fast_nb <= 1 << 17;
}

int fast_small_run(gts_index *idx, const int *d_qids, int qnum, int k, const int *d_carry, float *d_kth, int *d_ids,
                   float *d_dists, int **d_fail, int *n_fail, bool reset, cudaStream_t st)
{
    int rc = small_buffers(idx, st);
    if (rc) return rc;
    const FastShape fs = fast_shape(idx->dim);
    SmallArgs a{};
    a.t = idx->dev();
    a.bs = fast_summary(idx->fast_recs, fs, idx->fast_nb, idx->fast_nsb, idx->num);
    a.nb = idx->fast_nb;
    a.kp = fs.kp;
    a.qids = d_qids;
    a.qnum = qnum;
    a.k = k;
    while ((1 << a.jk) < k) a.jk++;
    a.carry = d_carry;
    int *c = (int *)idx->small_buf;
    a.nblk = c;
    a.ccnt = c + kSmallMax;
    a.ticket = c + 2 * kSmallMax;
    a.nfail = a.ticket + 1;
    a.fail = c + 256;
    a.blist = a.fail + kSmallMax;
    a.cpos = a.blist + (size_t)kSmallMax * idx->fast_nb;
    a.cv = (float *)(a.cpos + (size_t)kSmallMax * kSwCap);
    a.kth = d_kth;
    a.ids = d_ids;
    a.dists = d_dists;
    a.result = idx->small_result;
    a.stats = idx->d_stats;
    a.reset = reset ? 1 : 0;
    const int groups = (qnum + kSmGroup - 1) / kSmGroup;
    const dim3 pg(std::max(1, std::min((a.nb + 7) / 8, 8 * 148 / groups)), groups);
    const bool timed = idx->time_filter && idx->fev[0];   // the filter: everything before the exact values
    if (timed) GTS_CUDA_TRY(cudaEventRecord(idx->fev[0], st));
    if (fs.kp <= 64) k_small_prune<2><<<pg, 256, 0, st>>>(a);
    else if (fs.kp <= 128) k_small_prune<4><<<pg, 256, 0, st>>>(a);
    else k_small_prune<10><<<pg, 256, 0, st>>>(a);
    k_small_rows<<<dim3(std::max(8, 4 * 148 / qnum), qnum), 256, sizeof(float) * fs.kp, st>>>(a);
    if (timed) GTS_CUDA_TRY(cudaEventRecord(idx->fev[1], st));
    GTS_CUDA_TRY(cudaFuncSetAttribute(k_small_final, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinalSmem)));
    k_small_final<<<qnum, 128, sizeof(FinalSmem), st>>>(a);
    idx->kernel_launches += 3;
    GTS_CUDA_TRY(cudaGetLastError());
    GTS_CUDA_TRY(cudaStreamSynchronize(st));
    if (timed) {
        float ms = 0.f;
        GTS_CUDA_TRY(cudaEventElapsedTime(&ms, idx->fev[0], idx->fev[1]));
        idx->filter_ms += ms;
        idx->filter_launches++;
    }
    *n_fail = *(volatile int *)idx->small_result;
    *d_fail = a.fail;
    return GTS_OK;
}

}  // namespace gts
