// fast_order.cu -- the block order of the tensor-core kNN filter.
//
// The filter streams objects in blocks of up to 128 and skips a block for a
// tile of queries when the triangle inequality puts it out of every query's
// reach (|q - c| - radius > bound).  That only works when blocks are tight
// balls that never straddle two groups of the data.  A pivot-tree position
// order or a projection ball tree cut at fixed 128-object boundaries mixes
// groups in most blocks; here the order comes from a hierarchical k-means,
// built level by level on the device:
//
//   * a segment of more than kOrdHalve objects is split by Lloyd's k-means
//     into up to kOrdBranch children (about kOrdHalve objects each), so
//     well-separated groups never share a child;
//   * a segment of 129..kOrdHalve objects (or one k-means could not split)
//     is halved at a balanced point of its projection on the axis of a
//     2-means, so blocks come out nearly full;
//   * a segment of at most 128 objects is a block (padded to 128 slots).
//
// Every split is stable, so a segment keeps its position range for the rest
// of the build and the order nests: the first segment of at most kOrdSbMax
// objects on every path is a superblock, a contiguous run of blocks whose
// ball lets the filter drop all of them with one test.
//
// Per level: plan (k-means or halving), centroid seeds at evenly spread
// positions of the segment, kOrdIters Lloyd passes (one thread per object,
// sums per CTA, segment and child), a final
// pass that writes the sort key (segment, child) or (segment, projection),
// a stable radix sort, and the child segments.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cfloat>
#include <utility>
#include "fast.cuh"

namespace gts {

namespace {

constexpr int kOAsgPos = 256;         // positions (and threads) per assignment CTA
constexpr int kOAsgK = 16;            // dimensions per stage
constexpr int kOAsgLd = kOAsgK + 4;   // row stride in shared memory

__device__ __forceinline__ uint32_t order_bits(float f)
{
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void k_o_init(int n, int *perm, int *sid)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        perm[i] = i;
        sid[i] = 0;
    }
}

// kind: 0 leaf (<= 128 objects), 1 k-means split, 2 halving; kk: children.
__global__ void k_o_plan(int nseg, const int *__restrict__ sl, const int *__restrict__ sr,
                         const uint8_t *__restrict__ force, int *__restrict__ kind, int *__restrict__ kk,
                         int *__restrict__ active)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    const int size = sr[s] - sl[s];
    int kd = 0, K = 0;
    if (size > kFB) {
        if (force[s] || size <= kOrdHalve) {
            kd = 2;
            K = 2;
        } else {
            kd = 1;
            K = min(kOrdBranch, (size + kOrdHalve - 1) / kOrdHalve);
        }
        atomicAdd(active, 1);
    }
    kind[s] = kd;
    kk[s] = K;
}

__global__ void k_o_total(int nseg, const int *__restrict__ cbase, const int *__restrict__ kk, int *__restrict__ out)
{
    out[0] = cbase[nseg - 1] + kk[nseg - 1];
}

// One CTA per segment: seed its K centroids with the rows at positions
// l + (2j + 1) size / (2K).
__global__ void k_o_seed(int nseg, int dim, const float *__restrict__ rows, const int *__restrict__ perm,
                         const int *__restrict__ sl, const int *__restrict__ sr, const int *__restrict__ kk,
                         const int *__restrict__ cbase, float *__restrict__ cent)
{
    const int s = blockIdx.x;
    const int K = kk[s];
    if (K == 0) return;
    const int l = sl[s], size = sr[s] - l;
    for (int j = 0; j < K; j++) {
        const int p = l + (int)(((long long)(2 * j + 1) * size) / (2 * K));
        const float *x = rows + (size_t)perm[p] * dim;
        for (int d = threadIdx.x; d < dim; d += blockDim.x) cent[(size_t)(cbase[s] + j) * dim + d] = x[d];
    }
}

// Copies of 16 or 4 bytes to shared memory, zeros where !live.
__device__ __forceinline__ void cp_async16z(float *dst, const float *src, bool live)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async4z(float *dst, const float *src, bool live)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(live ? 4 : 0) : "memory");
}

struct alignas(16) AsgSmem {   // the centroids behind it are read 16 bytes at a time
    float x[2][kOAsgPos * kOAsgLd];   // staged dimensions of the positions' rows
    int row[kOAsgPos];                // their rows, later ordered by child
    int cnt[kOrdBranch], base[kOrdBranch + 1];
    // followed by the centroids, [dimensions rounded up to kOAsgK / 4][kOrdBranch][4]
};
static_assert(sizeof(AsgSmem) % 16 == 0, "centroids on a 16-byte boundary");

// acc[j] += squared differences of x and the KK centroids at c over the
// staged dimensions; the constant layout leaves no address arithmetic.
template <int KK>
__device__ __forceinline__ void dist_add(const float *x, const float *c, float (&acc)[kOrdBranch])
{
#pragma unroll
    for (int k = 0; k < kOAsgK; k += 4) {
        const float4 a = *reinterpret_cast<const float4 *>(x + k);
#pragma unroll
        for (int j = 0; j < KK; j++) {
            const float4 o = *reinterpret_cast<const float4 *>(c + k * kOrdBranch + 4 * j);
            const float e0 = a.x - o.x, e1 = a.y - o.y, e2 = a.z - o.z, e3 = a.w - o.w;
            acc[j] = fmaf(e3, e3, fmaf(e2, e2, fmaf(e1, e1, fmaf(e0, e0, acc[j]))));
        }
    }
}

// kOAsgPos consecutive positions per CTA, segment by segment.  Pass 0
// (Lloyd): nearest centroid of the segment, its sum and count.  Pass 1
// (final): the sort key (segment << 32 | child) for k-means segments,
// (segment << 32 | projection on c1 - c0) for halving segments, (segment
// << 32) for leaves; counts of the k-means children.
//
// A thread holds one position's distances to all centroids: the rows come 16
// dimensions at a time through shared memory (two stages, stride 20 floats,
// free of bank conflicts; the first 64 bytes bring 256 to L2), the centroids'
// reads are broadcasts.  The sums then read the rows again (from L2), ordered
// by child: a warp adds 32 dimensions of a child's rows in registers, one
// atomic addition each.  The rows' two reads (1 GB a pass at 1,000,000 x 128)
// and their latency bound it; four CTAs an SM hide more of it than three with
// more registers (11.1 against 11.8 ms over the 63 passes).  A pass there
// with 16 children takes 320 us and one with 2 200, the whole order 11.1 ms
// instead of 25.6 with a warp per position, bounded by 5 shuffles per position
// and child, and atomic additions per position in segments below 512.
// VEC: rows on 16-byte boundaries.
template <bool VEC>
__global__ void __launch_bounds__(kOAsgPos, 4) k_o_assign(int n, int dim, const float *__restrict__ rows,
                                                          const int *__restrict__ perm, const int *__restrict__ sid,
                                                          const int *__restrict__ sr, const int *__restrict__ kind,
                                                          const int *__restrict__ kk, const int *__restrict__ cbase,
                                                          const float *__restrict__ cent, float *__restrict__ csum,
                                                          int *__restrict__ ccnt, int final_pass,
                                                          unsigned long long *__restrict__ keys)
{
    extern __shared__ __align__(16) unsigned char asg_smem[];
    AsgSmem &sm = *reinterpret_cast<AsgSmem *>(asg_smem);
    const int nc = (dim + kOAsgK - 1) / kOAsgK, ldc = nc * kOAsgK;
    float *cs = reinterpret_cast<float *>(asg_smem + sizeof(AsgSmem));
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int p1 = min(n, (int)(blockIdx.x + 1) * kOAsgPos);
    for (int p = blockIdx.x * kOAsgPos, e; p < p1; p = e) {
        const int s = sid[p], kd = kind[s];
        e = min(p1, sr[s]);
        const int m = e - p;
        if (kd == 0) {
            if (final_pass && t < m) keys[p + t] = (unsigned long long)s << 32;
            continue;
        }
        const int K = kk[s], cb = cbase[s];
        const bool proj = final_pass && kd == 2;
        __syncthreads();   // the previous segment's reads are done
        if (t < m) sm.row[t] = perm[p + t];
        if (t < kOrdBranch) sm.cnt[t] = 0;
        for (int i = t; i < kOrdBranch * ldc; i += kOAsgPos) {
            const int j = i / ldc, d = i - j * ldc;
            float v = 0.f;
            if (d < dim && j < K) {
                v = cent[(size_t)(cb + j) * dim + d];
                if (proj && j == 0) v = cent[(size_t)(cb + 1) * dim + d] - v;
            }
            cs[(d >> 2) * (4 * kOrdBranch) + 4 * j + (d & 3)] = v;
        }
        __syncthreads();
        auto issue = [&](int ch) {
            float *dst = sm.x[ch & 1];
            const int k0 = ch * kOAsgK;
            if (VEC) {
#pragma unroll
                for (int u = 0; u < kOAsgK / 4; u++) {
                    const int i = t + u * kOAsgPos, r = i / (kOAsgK / 4), d = k0 + 4 * (i % (kOAsgK / 4));
                    if (r < m) {
                        const bool live = d < dim;
                        cp_async16z(dst + r * kOAsgLd + d - k0, rows + (size_t)sm.row[r] * dim + (live ? d : 0), live);
                    }
                }
            } else {
#pragma unroll 4
                for (int u = 0; u < kOAsgK; u++) {
                    const int i = t + u * kOAsgPos, r = i / kOAsgK, d = k0 + i % kOAsgK;
                    if (r < m) {
                        const bool live = d < dim;
                        cp_async4z(dst + r * kOAsgLd + d - k0, rows + (size_t)sm.row[r] * dim + (live ? d : 0), live);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float acc[kOrdBranch];
#pragma unroll
        for (int j = 0; j < kOrdBranch; j++) acc[j] = 0.f;
        issue(0);
        for (int ch = 0; ch < nc; ch++) {
            // the stage has come, and everyone is done with the other one
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (ch + 1 < nc) issue(ch + 1);
            if (warp * 32 >= m) continue;
            const float *x = sm.x[ch & 1] + t * kOAsgLd, *c = cs + ch * (kOAsgK * kOrdBranch);
            if (proj) {
#pragma unroll
                for (int k = 0; k < kOAsgK; k += 4) {
                    const float4 a = *reinterpret_cast<const float4 *>(x + k);
                    const float4 o = *reinterpret_cast<const float4 *>(c + k * kOrdBranch);
                    acc[0] = fmaf(a.w, o.w, fmaf(a.z, o.z, fmaf(a.y, o.y, fmaf(a.x, o.x, acc[0]))));
                }
            } else if (K <= 2) {
                dist_add<2>(x, c, acc);
            } else if (K <= 4) {
                dist_add<4>(x, c, acc);
            } else if (K <= 8) {
                dist_add<8>(x, c, acc);
            } else {
                dist_add<kOrdBranch>(x, c, acc);
            }
        }
        if (proj) {
            if (t < m) keys[p + t] = ((unsigned long long)s << 32) | order_bits(acc[0]);
            continue;
        }
        int bj = 0, at = 0;
        float best = FLT_MAX;
#pragma unroll
        for (int j = 0; j < kOrdBranch; j++)
            if (j < K && acc[j] < best) {
                best = acc[j];
                bj = j;
            }
        const int row = t < m ? sm.row[t] : 0;
        if (t < m) at = atomicAdd(&sm.cnt[bj], 1);
        __syncthreads();
        if (t < K && sm.cnt[t]) atomicAdd(&ccnt[cb + t], sm.cnt[t]);
        if (final_pass) {
            if (t < m) keys[p + t] = ((unsigned long long)s << 32) | (uint32_t)bj;
            continue;
        }
        if (t <= kOrdBranch) {
            int b = 0;
            for (int j = 0; j < t; j++) b += sm.cnt[j];
            sm.base[t] = b;
        }
        __syncthreads();
        if (t < m) sm.row[sm.base[bj] + at] = row;
        __syncthreads();
        const int ng = (dim + 31) / 32;
        for (int task = warp; task < 2 * ng; task += kOAsgPos / 32) {
            const int d = (task >> 1) * 32 + lane, i0 = task & 1 ? m / 2 : 0, i1 = task & 1 ? m : m / 2;
            for (int j = 0; j < K; j++) {
                const int lo = max(sm.base[j], i0), hi = min(sm.base[j + 1], i1);
                if (lo >= hi || d >= dim) continue;
                float v = 0.f;
#pragma unroll 8
                for (int i = lo; i < hi; i++) v += rows[(size_t)sm.row[i] * dim + d];
                atomicAdd(&csum[(size_t)(cb + j) * dim + d], v);
            }
        }
    }
}

__global__ void k_o_update(int C, int dim, const float *__restrict__ csum, const int *__restrict__ ccnt,
                           float *__restrict__ cent)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)C * dim) return;
    const int c = (int)(i / dim);
    if (ccnt[c] > 0) cent[i] = csum[i] / (float)ccnt[c];
}

__global__ void k_o_nchild(int nseg, const int *__restrict__ kind, const int *__restrict__ kk,
                           const int *__restrict__ cbase, const int *__restrict__ ccnt, int *__restrict__ nchild)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    int c = 1;
    if (kind[s] == 2) c = 2;
    else if (kind[s] == 1) {
        c = 0;
        for (int j = 0; j < kk[s]; j++) c += ccnt[cbase[s] + j] > 0;
    }
    nchild[s] = c;
}

// Child segments of every segment, at newbase[s]; superblock starts where a
// segment of more than kOrdSbMax objects has a child of at most kOrdSbMax.
__global__ void k_o_children(int nseg, const int *__restrict__ sl, const int *__restrict__ sr,
                             const int *__restrict__ kind, const int *__restrict__ kk, const int *__restrict__ cbase,
                             const int *__restrict__ ccnt, const int *__restrict__ newbase, int *__restrict__ nsl,
                             int *__restrict__ nsr, uint8_t *__restrict__ nforce, uint8_t *__restrict__ sb_start)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    const int l = sl[s], r = sr[s], size = r - l, b = newbase[s];
    const bool big = size > kOrdSbMax;
    if (kind[s] == 0) {
        nsl[b] = l;
        nsr[b] = r;
        nforce[b] = 0;
    } else if (kind[s] == 1) {
        const int cb = cbase[s], K = kk[s];
        int nz = 0;
        for (int j = 0; j < K; j++) nz += ccnt[cb + j] > 0;
        int run = l, c = 0;
        for (int j = 0; j < K; j++) {
            const int cnt = ccnt[cb + j];
            if (cnt == 0) continue;
            nsl[b + c] = run;
            nsr[b + c] = run + cnt;
            nforce[b + c] = nz == 1;   // k-means could not split it: halve next
            if (big && cnt <= kOrdSbMax) sb_start[run] = 1;
            run += cnt;
            c++;
        }
    } else {
        const int nbk = (size + kFB - 1) / kFB;
        const int m = l + (int)(((long long)size * ((nbk + 1) / 2)) / nbk);
        nsl[b] = l;
        nsr[b] = m;
        nsl[b + 1] = m;
        nsr[b + 1] = r;
        nforce[b] = nforce[b + 1] = 0;
        if (big && m - l <= kOrdSbMax) sb_start[l] = 1;
        if (big && r - m <= kOrdSbMax) sb_start[m] = 1;
    }
}

__global__ void k_o_relabel(int n, int *__restrict__ sid, const int *__restrict__ newbase,
                            const int *__restrict__ nchild, const int *__restrict__ nsl)
{
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= n) return;
    const int s = sid[pos], b = newbase[s], c = nchild[s];
    int j = 0;
    while (j + 1 < c && nsl[b + j + 1] <= pos) j++;
    sid[pos] = b + j;
}

// Superblock of every block: flags f[b] = sb_start[blk_l[b]].
__global__ void k_o_sbflag(int nb, const int *__restrict__ bl, const uint8_t *__restrict__ sb_start,
                           int *__restrict__ f)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < nb) f[b] = sb_start[bl[b]] ? 1 : 0;
}

__global__ void k_o_sbtable(int nb, const int *__restrict__ f, const int *__restrict__ incl, int *__restrict__ blk_sb,
                            int *__restrict__ sb_b0, int *__restrict__ nsb_out)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    blk_sb[b] = incl[b] - 1;
    if (f[b]) sb_b0[incl[b] - 1] = b;
    if (b == nb - 1) {
        sb_b0[incl[b]] = nb;
        *nsb_out = incl[b];
    }
}

}  // namespace

int fast_block_order(gts_index *idx, FastOrder *out, cudaStream_t st)
{
    const int n = idx->num, dim = idx->dim;
    if (n < 1 || dim > kFMaxKp) {
        gts_set_error("block order: %d objects of dimension %d (at most %d)", n, dim, kFMaxKp);
        return GTS_ERR_INVALID;
    }
    const int S = n + 1;                        // segments (each holds at least one object)
    const int Ccap = n / 32 + 4 * kOrdBranch;   // centroids: <= 16 per k-means segment (> kOrdHalve objects)
                                                // plus 2 per halving segment (> 128 objects)
    size_t cub_bytes = 0, tb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (unsigned long long *)nullptr, (unsigned long long *)nullptr,
                                    (int *)nullptr, (int *)nullptr, n, 0, 64, st);
    cub_bytes = tb;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, (int *)nullptr, (int *)nullptr, S, st);
    cub_bytes = std::max(cub_bytes, tb);
    cub::DeviceScan::InclusiveSum(nullptr, tb, (int *)nullptr, (int *)nullptr, S, st);
    cub_bytes = std::max(cub_bytes, tb);

    size_t off = 0;
    auto take = [&](size_t b) { size_t o = off; off += (b + 255) & ~(size_t)255; return o; };
    const size_t o_perm = take(4 * (size_t)n), o_perm2 = take(4 * (size_t)n), o_sid = take(4 * (size_t)n);
    const size_t o_keys = take(8 * (size_t)n), o_keys2 = take(8 * (size_t)n);
    size_t o_seg[11];
    for (int i = 0; i < 11; i++) o_seg[i] = take(4 * (size_t)S);
    const size_t o_force = take(S), o_nforce = take(S), o_sbs = take((size_t)n);
    const size_t o_cent = take(4 * (size_t)Ccap * dim), o_csum = take(4 * (size_t)Ccap * dim);
    const size_t o_ccnt = take(4 * (size_t)Ccap), o_misc = take(64), o_cub = take(cub_bytes);
    int rc;
    if ((rc = ensure_scratch(idx, off))) return rc;
    unsigned char *B = (unsigned char *)idx->scratch;
    int *perm = (int *)(B + o_perm), *perm2 = (int *)(B + o_perm2), *sid = (int *)(B + o_sid);
    unsigned long long *keys = (unsigned long long *)(B + o_keys), *keys2 = (unsigned long long *)(B + o_keys2);
    int *sl = (int *)(B + o_seg[0]), *sr = (int *)(B + o_seg[1]), *nsl = (int *)(B + o_seg[2]);
    int *nsr = (int *)(B + o_seg[3]), *kind = (int *)(B + o_seg[4]), *kk = (int *)(B + o_seg[5]);
    int *cbase = (int *)(B + o_seg[6]), *nchild = (int *)(B + o_seg[7]), *newbase = (int *)(B + o_seg[8]);
    int *flag = (int *)(B + o_seg[9]), *incl = (int *)(B + o_seg[10]);
    uint8_t *force = B + o_force, *nforce = B + o_nforce, *sb_start = B + o_sbs;
    float *cent = (float *)(B + o_cent), *csum = (float *)(B + o_csum);
    int *ccnt = (int *)(B + o_ccnt), *misc = (int *)(B + o_misc);
    void *cub_tmp = B + o_cub;

    k_o_init<<<(n + 255) / 256, 256, 0, st>>>(n, perm, sid);
    const int h_seg[2] = {0, n};
    GTS_CUDA_TRY(cudaMemcpyAsync(sl, &h_seg[0], sizeof(int), cudaMemcpyHostToDevice, st));
    GTS_CUDA_TRY(cudaMemcpyAsync(sr, &h_seg[1], sizeof(int), cudaMemcpyHostToDevice, st));
    GTS_CUDA_TRY(cudaMemsetAsync(force, 0, 1, st));
    GTS_CUDA_TRY(cudaMemsetAsync(sb_start, 0, (size_t)n, st));
    if (n <= kOrdSbMax) GTS_CUDA_TRY(cudaMemsetAsync(sb_start, 1, 1, st));
    int nseg = 1, level = 0;
    const int agrid = (n + kOAsgPos - 1) / kOAsgPos;
    const bool vec = dim % 4 == 0 && (uintptr_t)idx->rows % 16 == 0;
    const size_t asmem = sizeof(AsgSmem) + sizeof(float) * kOrdBranch * ((dim + kOAsgK - 1) / kOAsgK * kOAsgK);
    auto assign_fn = vec ? k_o_assign<true> : k_o_assign<false>;
    GTS_CUDA_TRY(cudaFuncSetAttribute(assign_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)asmem));
    auto assign = [&](int final_pass) {
        assign_fn<<<agrid, kOAsgPos, asmem, st>>>(n, dim, idx->rows, perm, sid, sr, kind, kk, cbase, cent, csum, ccnt,
                                                  final_pass, keys);
        GTS_CUDA_TRY(cudaGetLastError());
        return (int)GTS_OK;
    };
    for (; level < kOrdMaxLevels; level++) {
        GTS_CUDA_TRY(cudaMemsetAsync(misc, 0, 2 * sizeof(int), st));
        k_o_plan<<<(nseg + 255) / 256, 256, 0, st>>>(nseg, sl, sr, force, kind, kk, misc);
        size_t tb2 = cub_bytes;
        GTS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, tb2, kk, cbase, nseg, st));
        k_o_total<<<1, 1, 0, st>>>(nseg, cbase, kk, misc + 1);
        int h[2];
        GTS_CUDA_TRY(cudaMemcpyAsync(h, misc, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
        GTS_CUDA_TRY(cudaStreamSynchronize(st));
        const int active = h[0], C = h[1];
        if (active == 0) break;
        if (C > Ccap) {
            gts_set_error("block order: %d centroids exceed the capacity %d", C, Ccap);
            return GTS_ERR_KERNEL;
        }
        k_o_seed<<<nseg, 128, 0, st>>>(nseg, dim, idx->rows, perm, sl, sr, kk, cbase, cent);
        const int ugrid = (int)(((size_t)C * dim + 255) / 256);
        for (int it = 0; it < kOrdIters; it++) {
            GTS_CUDA_TRY(cudaMemsetAsync(csum, 0, sizeof(float) * (size_t)C * dim, st));
            GTS_CUDA_TRY(cudaMemsetAsync(ccnt, 0, sizeof(int) * (size_t)C, st));
            if ((rc = assign(0))) return rc;
            k_o_update<<<ugrid, 256, 0, st>>>(C, dim, csum, ccnt, cent);
        }
        GTS_CUDA_TRY(cudaMemsetAsync(ccnt, 0, sizeof(int) * (size_t)C, st));
        if ((rc = assign(1))) return rc;
        int sbits = 1;
        while ((1 << sbits) < nseg) sbits++;
        size_t tb3 = cub_bytes;
        GTS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(cub_tmp, tb3, keys, keys2, perm, perm2, n, 0, 32 + sbits, st));
        std::swap(perm, perm2);
        k_o_nchild<<<(nseg + 255) / 256, 256, 0, st>>>(nseg, kind, kk, cbase, ccnt, nchild);
        size_t tb4 = cub_bytes;
        GTS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, tb4, nchild, newbase, nseg, st));
        k_o_total<<<1, 1, 0, st>>>(nseg, newbase, nchild, misc);
        k_o_children<<<(nseg + 255) / 256, 256, 0, st>>>(nseg, sl, sr, kind, kk, cbase, ccnt, newbase, nsl, nsr,
                                                         nforce, sb_start);
        k_o_relabel<<<(n + 255) / 256, 256, 0, st>>>(n, sid, newbase, nchild, nsl);
        GTS_CUDA_TRY(cudaGetLastError());
        int total = 0;
        GTS_CUDA_TRY(cudaMemcpyAsync(&total, misc, sizeof(int), cudaMemcpyDeviceToHost, st));
        GTS_CUDA_TRY(cudaStreamSynchronize(st));
        if (total < nseg || total > S) {
            gts_set_error("block order: level %d produced %d segments from %d", level, total, nseg);
            return GTS_ERR_KERNEL;
        }
        nseg = total;
        std::swap(sl, nsl);
        std::swap(sr, nsr);
        std::swap(force, nforce);
    }
    if (level == kOrdMaxLevels) {
        gts_set_error("block order: no convergence after %d levels", kOrdMaxLevels);
        return GTS_ERR_KERNEL;
    }
    // blocks = the final segments; superblocks from the recorded starts
    const int nb = nseg;
    int *blk_sb = nchild, *sb_b0 = newbase;   // reuse (segment-sized arrays)
    k_o_sbflag<<<(nb + 255) / 256, 256, 0, st>>>(nb, sl, sb_start, flag);
    size_t tb5 = cub_bytes;
    GTS_CUDA_TRY(cub::DeviceScan::InclusiveSum(cub_tmp, tb5, flag, incl, nb, st));
    k_o_sbtable<<<(nb + 255) / 256, 256, 0, st>>>(nb, flag, incl, blk_sb, sb_b0, misc);
    GTS_CUDA_TRY(cudaGetLastError());
    int nsb = 0;
    GTS_CUDA_TRY(cudaMemcpyAsync(&nsb, misc, sizeof(int), cudaMemcpyDeviceToHost, st));
    GTS_CUDA_TRY(cudaStreamSynchronize(st));
    if (nsb < 1 || nsb > nb) {
        gts_set_error("block order: %d superblocks for %d blocks", nsb, nb);
        return GTS_ERR_KERNEL;
    }
    out->nb = nb;
    out->nsb = nsb;
    out->perm = perm;
    out->blk_l = sl;
    out->blk_r = sr;
    out->blk_sb = blk_sb;
    out->sb_b0 = sb_b0;
    return GTS_OK;
}

}  // namespace gts
