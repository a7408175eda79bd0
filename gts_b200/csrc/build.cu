// build.cu -- parallel pivot-tree construction on the device.
//
// Restates indexConstru (tree.cuh:332-393) level by level:
//   1. k_select_pivots: for every node split at this level the pivot is the
//      object at the middle rank of the node's range, id_list[(lid+rid)/2]
//      (tree.cuh:73), and the node's range becomes one sort segment;
//   2. k_keys: every object of a split node gets the reference's double key
//      dist/INFI_DIS + b*DIS_CODE (tree.cuh:155), distance in the
//      F64-accumulated build arithmetic;
//   3. a stable sort of (key, id) inside each split node: one radix sort of
//      all keys, then (below the root) one by the node's first position, so
//      every node's range keeps its place and an unsplit node its order (eight
//      plus a few radix passes over the whole chip; a segmented sort gave each
//      of the few huge segments near the root one CTA: 19.2 ms against 1.9 for
//      the five levels of 1,000,000 objects; small indexes keep it, done
//      before a radix sort's dozen passes: building 5,000 x 8 takes 1.00 ms by
//      segments and 1.30 by radix, 12,000 x 32 1.8 and 1.3).  The reference
//      sorts all N keys globally (tree.cuh:372); node codes keep the segments
//      apart and the sort is stable, so for every tree in which each level's
//      objects all sit in split nodes the order is identical;
//   4. k_split: O children per split node with the equal-count split, the
//      last child taking the remainder, min_dis = dist(first object of the
//      child, pivot) in F32-accumulated arithmetic, is_leaf = size <= MAX_SIZE
//      (tree.cuh:191-295);
//   5. k_node_of_pos: each position learns its child, so the next level can
//      run one thread per object instead of one block per node.
// One 4-byte device->host read per level (the number of nodes still to
// split) decides whether to continue, as the reference's reduce does.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_segmented_sort.cuh>
#include <cstdio>
#include <vector>
#include "index.cuh"

namespace gts {

template <typename T>
int dev_alloc(T **p, size_t n, size_t *acct)
{
    *p = nullptr;
    if (n == 0) n = 1;
    cudaError_t e = dev_malloc((void **)p, n * sizeof(T));
    if (e != cudaSuccess) {
        cudaGetLastError();
        gts_set_error("cudaMalloc of %zu bytes failed: %s", n * sizeof(T), cudaGetErrorString(e));
        return GTS_ERR_NOMEM;
    }
    if (acct) *acct += n * sizeof(T);
    return GTS_OK;
}
template int dev_alloc<float>(float **, size_t, size_t *);
template int dev_alloc<int>(int **, size_t, size_t *);
template int dev_alloc<char>(char **, size_t, size_t *);
template int dev_alloc<uint8_t>(uint8_t **, size_t, size_t *);
template int dev_alloc<double>(double **, size_t, size_t *);
template int dev_alloc<uint32_t>(uint32_t **, size_t, size_t *);
template int dev_alloc<unsigned short>(unsigned short **, size_t, size_t *);
template int dev_alloc<unsigned long long>(unsigned long long **, size_t, size_t *);
template int dev_alloc<int4>(int4 **, size_t, size_t *);
template int dev_alloc<uint4>(uint4 **, size_t, size_t *);

// Build-time distance between two objects (by id), F64 or F32 site.
__device__ __forceinline__ double obj_dist(const DevData &d, int a, int b, int acc)
{
    if (d.metric == kEdit) {
        return (double)edit_dp(d.strs + (size_t)a * kStrStride, d.lens[a],
                               d.strs + (size_t)b * kStrStride, d.lens[b]);
    }
    const float *x = d.rows + (size_t)a * d.dim;
    const float *y = d.rows + (size_t)b * d.dim;
    if (acc == kAccF64) return dist_row_f64(x, y, d.dim, d.metric);
    if (d.metric == kL2) {
        float r = 0.f;
#pragma unroll 8
        for (int j = 0; j < d.dim; j++) r = add_square(r, x[j] - y[j]);
        return (double)(float)pow(r, 0.5);
    }
    return (double)dist_row_f32(x, y, d.dim, d.metric);
}

__global__ void k_init(int n, int mnn, int *id_list, int *node_of_pos, int *node_pid,
                       int *node_size, int *node_lid, int *node_pivot, float *node_min_dis,
                       uint8_t *node_flags, uint8_t *split)
{
    size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = tid; i < (size_t)n; i += stride) {
        id_list[i] = (int)i;
        node_of_pos[i] = 0;
    }
    for (size_t i = tid; i < (size_t)mnn; i += stride) {
        node_pid[i] = -1;
        node_size[i] = 0;
        node_lid[i] = 0;
        node_pivot[i] = -1;
        node_min_dis[i] = 0.f;
        node_flags[i] = 0;
        split[i] = 0;
    }
    if (tid == 0) {   // initIndexData (tree.cuh:308-317)
        node_size[0] = n;
        node_lid[0] = 0;
        node_pid[0] = -1;
        node_min_dis[0] = 0.f;
        node_flags[0] = kExists;
        split[0] = 1;
    }
}

// seg (nullable): [2][nb] the nodes' ranges as sort segments, empty for those not split.
__global__ void k_select_pivots(int start, int nb, const int *id_list, const int *node_size,
                                const int *node_lid, const uint8_t *split, int *node_pivot, int *seg)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    int nid = start + b;
    if (seg) {
        seg[b] = split[nid] ? node_lid[nid] : 0;
        seg[nb + b] = split[nid] ? node_lid[nid] + node_size[nid] : 0;
    }
    if (split[nid]) {
        int lid = node_lid[nid], size = node_size[nid];
        int rid = lid + size - 1;
        node_pivot[nid] = id_list[(lid + rid) / 2];
    }
}

__global__ void k_keys(DevData d, int n, int start, int nb, int dis_code, int infi_dis,
                       const int *id_list, const int *node_of_pos, const uint8_t *split,
                       const int *node_pivot, double *key, int *posv)
{
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t pos = (size_t)blockIdx.x * blockDim.x + threadIdx.x; pos < (size_t)n; pos += stride) {
        int nid = node_of_pos[pos];
        int b = nid - start;
        posv[pos] = (int)pos;
        key[pos] = 0.0;   // an unsplit node keeps its order
        if (b < 0 || b >= nb || !split[nid]) continue;
        double res = obj_dist(d, id_list[pos], node_pivot[nid], kAccF64);
        key[pos] = (double)(res / infi_dis + b * dis_code);
    }
}

// Sort key of the second pass: the first position of the node that holds
// the object (node ranges partition the positions in order).
__global__ void k_node_lids(int n, const int *posv, const int *node_of_pos, const int *node_lid, uint32_t *lid)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) lid[i] = (uint32_t)node_lid[node_of_pos[posv[i]]];
}

__global__ void k_apply_order(int n, const int *posv, const int *ids, int *out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = ids[posv[i]];
}

// A thread per child; its one distance is a chain of dim dependent steps, in
// FP32 where pow would take 600 cycles of the chip's FP64 each (add_square):
// 184 -> 72 us a level at 300 dimensions.
__global__ void k_split(DevData d, int start, int nb, int order, int max_size, const int *id_list,
                        const uint8_t *split_in, int *node_pid, int *node_size, int *node_lid,
                        const int *node_pivot, float *node_min_dis, uint8_t *node_flags,
                        uint8_t *split, int *nsplit)
{
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)nb * order) return;
    int b = (int)(t / order), i = (int)(t % order);
    int nid = start + b;
    if (!split_in[nid]) return;
    int lid = node_lid[nid], size = node_size[nid];
    int avg = size / order;
    long c = (long)nid * order + i + 1;
    int clid = lid + avg * i;
    int csize = (i < order - 1) ? avg : size - (order - 1) * avg;
    int piv = node_pivot[nid];
    node_lid[c] = clid;
    node_pid[c] = piv;
    node_size[c] = csize;
    node_min_dis[c] = (float)obj_dist(d, id_list[clid], piv, kAccF32);
    bool leaf = csize <= max_size;
    node_flags[c] = kExists | (leaf ? kLeaf : 0);
    split[c] = leaf ? 0 : 1;
    if (!leaf) atomicAdd(nsplit, 1);
}

__global__ void k_node_of_pos(int n, int start, int nb, int order, const uint8_t *split,
                              const int *node_size, const int *node_lid, int *node_of_pos)
{
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t pos = (size_t)blockIdx.x * blockDim.x + threadIdx.x; pos < (size_t)n; pos += stride) {
        int nid = node_of_pos[pos];
        int b = nid - start;
        if (b < 0 || b >= nb || !split[nid]) continue;
        int avg = node_size[nid] / order;
        int off = (int)pos - node_lid[nid];
        int ci = avg > 0 ? min(off / avg, order - 1) : order - 1;
        node_of_pos[pos] = nid * order + 1 + ci;
    }
}

__global__ void k_clear_level(int start, int nb, uint8_t *split)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < nb) split[start + b] = 0;
}

// Tree-order copies of the data so that a leaf's objects are contiguous.
// Character-class signatures of the strings in tree order (edit lower bounds)
// and their first kPackChars characters (zeros past the end) as two 16-byte words.
// In lens: characters altogether, strings of more than 32 and of more than 64.
__global__ void k_str_sig(int n, const char *tstrs, const int *tlens, uint4 *tsig, uint4 *tpack, unsigned long long *lens)
{
    unsigned chars = 0, over32 = 0, over64 = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)n; i += (size_t)gridDim.x * blockDim.x) {
        const char *s = tstrs + i * kStrStride;
        const int len = tlens[i];
        tsig[i] = str_sig(s, len);
        chars += max(len, 0);
        over32 += len > 32;
        over64 += len > 64;
        uint32_t w[kPackChars / 4];
#pragma unroll
        for (int k = 0; k < kPackChars / 4; k++) {
            uint32_t v = 0;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (4 * k + j < len) v |= (uint32_t)(unsigned char)s[4 * k + j] << (8 * j);
            w[k] = v;
        }
        tpack[2 * i] = make_uint4(w[0], w[1], w[2], w[3]);
        tpack[2 * i + 1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    chars = __reduce_add_sync(0xffffffffu, chars);
    over32 = __reduce_add_sync(0xffffffffu, over32);
    over64 = __reduce_add_sync(0xffffffffu, over64);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&lens[0], (unsigned long long)chars);
        atomicAdd(&lens[1], (unsigned long long)over32);
        atomicAdd(&lens[2], (unsigned long long)over64);
    }
}

__global__ void k_permute(int n, int dim, int metric, const int *id_list, const float *rows,
                          float *trows, const char *strs, char *tstrs, const int *lens, int *tlens,
                          int *pos_of_id)
{
    size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (metric == kEdit) {
        for (size_t i = tid; i < (size_t)n * kStrStride; i += stride) {
            size_t pos = i / kStrStride, c = i % kStrStride;
            tstrs[i] = strs[(size_t)id_list[pos] * kStrStride + c];
        }
    } else {
        for (size_t i = tid; i < (size_t)n * dim; i += stride) {
            size_t pos = i / dim, c = i % dim;
            trows[i] = rows[(size_t)id_list[pos] * dim + c];
        }
    }
    for (size_t pos = tid; pos < (size_t)n; pos += stride) {
        int id = id_list[pos];
        pos_of_id[id] = (int)pos;
        if (metric == kEdit) tlens[pos] = lens[id];
    }
}

// The nodes as records, and the batched sweep's cut nodes, in pieces of at most
// kCutSize objects, and their ancestors (index.cuh); a CTA appends its nodes
// in order, so lists stay nearly in position order.  Also the number of
// childless nodes, counts[2].
__global__ void __launch_bounds__(256) k_cut_lists(int mnn, int order, const uint8_t *flags, const int *size,
                                                   const int *pivot, const int *lid, const float *min_dis, int2 *cut,
                                                   int *anc, int *anc_idx, int *counts, int4 *rec)
{
    __shared__ int base[2], woff[2][8];
    const int i = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool inner = false;
    int pieces = 0;
    const int leaves = __syncthreads_count(i < mnn && (flags[i] & kExists) && size[i] > 0 && pivot[i] < 0);
    if (threadIdx.x == 0 && leaves) atomicAdd(&counts[2], leaves);
    // a child that does not exist still bounds its neighbour's ring by its min_dis (0)
    if (i < mnn) rec[i] = make_int4(__float_as_int(min_dis[i]), (flags[i] & kExists) ? size[i] : 0, lid[i], pivot[i]);
    if (i < mnn && (flags[i] & kExists) && size[i] > 0) {
        inner = pivot[i] >= 0 && size[i] > kCutSize;
        if (!inner && (i == 0 || size[(i - 1) / order] > kCutSize)) pieces = (size[i] + kCutSize - 1) / kCutSize;
    }
    const unsigned m = __ballot_sync(0xffffffffu, inner);
    int incl = pieces;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) woff[0][warp] = incl;
    if (lane == 0) woff[1][warp] = __popc(m);
    __syncthreads();
    if (threadIdx.x < 2) {
        const int u = threadIdx.x;
        int run = 0;
        for (int w = 0; w < 8; w++) {
            const int c = woff[u][w];
            woff[u][w] = run;
            run += c;
        }
        base[u] = run ? atomicAdd(&counts[u], run) : 0;
    }
    __syncthreads();
    if (inner) {
        const int at = base[1] + woff[1][warp] + __popc(m & ((1u << lane) - 1u));
        anc[at] = i;
        anc_idx[i] = at;
    }
    const int at = base[0] + woff[0][warp] + incl - pieces;
    if (pieces == 1) cut[at] = make_int2(i, 0);
    for (unsigned todo = __ballot_sync(0xffffffffu, pieces > 1); todo; todo &= todo - 1) {   // a large leaf: the warp together
        const int from = __ffs(todo) - 1, node = __shfl_sync(0xffffffffu, i, from);
        const int n = __shfl_sync(0xffffffffu, pieces, from), o = __shfl_sync(0xffffffffu, at, from);
        for (int j = lane; j < n; j += 32) cut[o + j] = make_int2(node, j * kCutSize);
    }
}

// Norms of the rows in tree order, in the angle metric's own arithmetic
// (dist_row_f64): FP32 fused sums in dimension order.
__global__ void k_row_norms(int n, int dim, const float *trows, float *tnorm)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)n; i += (size_t)gridDim.x * blockDim.x) {
        const float *a = trows + i * dim;
        float sa = 0.f;
        for (int j = 0; j < dim; j++) sa = fmaf(a[j], a[j], sa);
        sa = pow(sa, 0.5);
        tnorm[i] = sa;
    }
}

static inline unsigned grid_for(size_t n, int block, unsigned cap = 148u * 32u)
{
    size_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    return (unsigned)(g > cap ? cap : g);
}

constexpr int kSegSortMax = 8192;   // objects up to which a level is sorted by segments

int ensure_scratch(gts_index *idx, size_t bytes)
{
    if (idx->scratch_bytes >= bytes) return GTS_OK;
    if (idx->scratch) dev_free(idx->scratch);
    idx->scratch = nullptr;
    idx->scratch_bytes = 0;
    if (dev_malloc(&idx->scratch, bytes) != cudaSuccess) {
        cudaGetLastError();
        idx->scratch = nullptr;
        gts_set_error("cudaMalloc of %zu bytes of search scratch failed", bytes);
        return GTS_ERR_NOMEM;
    }
    idx->scratch_bytes = bytes;
    return GTS_OK;
}

int ensure_io(gts_index *idx, size_t bytes)
{
    if (bytes <= idx->io_bytes) return GTS_OK;
    if (idx->io) dev_free(idx->io);
    idx->io = nullptr;
    idx->io_bytes = 0;
    size_t want = bytes + bytes / 4 + 4096;
    if (dev_malloc(&idx->io, want) != cudaSuccess) {
        cudaGetLastError();
        idx->io = nullptr;
        gts_set_error("cudaMalloc of %zu bytes of argument buffers failed", want);
        return GTS_ERR_NOMEM;
    }
    idx->io_bytes = want;
    return GTS_OK;
}

int ensure_hits(gts_index *idx, size_t bytes, size_t room, void **out)
{
    if (bytes > idx->hits_bytes) {
        if (idx->hits) dev_free(idx->hits);
        idx->hits = nullptr;
        idx->hits_bytes = 0;
        const size_t want = std::max(bytes, std::min(bytes + bytes / 4, room));
        if (dev_malloc(&idx->hits, want) != cudaSuccess) {
            cudaGetLastError();
            idx->hits = nullptr;
            gts_set_error("cudaMalloc of %zu bytes for the hits failed", want);
            return GTS_ERR_NOMEM;
        }
        idx->hits_bytes = want;
    }
    *out = idx->hits;
    return GTS_OK;
}

void free_tree(gts_index *idx)
{
    if (idx->fast_recs) dev_free(idx->fast_recs);
    idx->fast_recs = nullptr;
    idx->fast_nb = 0;
    idx->fast_nsb = 0;
    for (int &c : idx->fast_cfg) c = 0;
    for (bool &b : idx->fast_pinned) b = false;
    for (int &c : idx->plain_nt) c = 0;
    for (bool &b : idx->plain_pinned) b = false;
    for (bool &b : idx->plain_passed) b = false;
    graph_invalidate(idx);
    idx->mlp_ready = false;   // its feature pivots belong to the old tree
    void *ps[] = {idx->trows, idx->tstrs, idx->tlens, idx->tsig, idx->tpack, idx->id_list, idx->pos_of_id, idx->node_pid,
                  idx->node_size, idx->node_lid, idx->node_pivot, idx->node_min_dis,
                  idx->node_flags, idx->cut_node, idx->cut_anc, idx->cut_anc_idx, idx->tnorm, idx->node_rec};
    for (void *p : ps)
        if (p) dev_free(p);
    idx->trows = nullptr; idx->tstrs = nullptr; idx->tlens = nullptr; idx->tsig = nullptr; idx->tpack = nullptr;
    idx->id_list = nullptr; idx->pos_of_id = nullptr; idx->node_pid = nullptr;
    idx->node_size = nullptr; idx->node_lid = nullptr; idx->node_pivot = nullptr;
    idx->node_min_dis = nullptr; idx->node_flags = nullptr;
    idx->cut_node = nullptr; idx->cut_anc = nullptr; idx->cut_anc_idx = nullptr; idx->tnorm = nullptr;
    idx->node_rec = nullptr;
    idx->ncut = idx->ncut_anc = idx->nleaf = 0;
}

void free_data(gts_index *idx)
{
    graph_invalidate(idx);   // the captured filter pass reads the rows
    if (idx->rows) dev_free(idx->rows);
    if (idx->strs) dev_free(idx->strs);
    if (idx->lens) dev_free(idx->lens);
    idx->rows = nullptr; idx->strs = nullptr; idx->lens = nullptr;
}

namespace {
// Build-time scratch, released on every exit path.
struct BuildScratch {
    int *node_of_pos = nullptr, *ids_alt = nullptr, *posv = nullptr, *posv_alt = nullptr, *nsplit = nullptr, *seg = nullptr;
    double *key = nullptr, *key_alt = nullptr;
    uint8_t *split = nullptr;
    unsigned long long *lens = nullptr;
    void *temp = nullptr;
    ~BuildScratch()
    {
        void *ps[] = {node_of_pos, ids_alt, posv, posv_alt, nsplit, seg, key, key_alt, split, lens, temp};
        for (void *p : ps)
            if (p) dev_free(p);
    }
};
}  // namespace

static int build_tree_impl(gts_index *idx, cudaStream_t s)
{
    const gts_params &p = idx->params;
    const int n = idx->num, O = p.tree_order, H = p.max_h;
    double mnn_d = (pow((double)O, (double)H) - 1) / (O - 1);   // tree.cuh:339
    if (mnn_d > 2.0e9) {
        gts_set_error("max_node_num too large (order %d, max_h %d)", O, H);
        return GTS_ERR_INVALID;
    }
    const int mnn = (int)mnn_d;
    idx->max_node_num = mnn;

    size_t acct = 0;
    int rc;
#define ALLOC(ptr, cnt) \
    if ((rc = dev_alloc(&(ptr), (cnt), &acct)) != GTS_OK) return rc;
    ALLOC(idx->id_list, n);
    ALLOC(idx->pos_of_id, n);
    ALLOC(idx->node_pid, mnn);
    ALLOC(idx->node_size, mnn);
    ALLOC(idx->node_lid, mnn);
    ALLOC(idx->node_pivot, mnn);
    ALLOC(idx->node_min_dis, mnn);
    ALLOC(idx->node_flags, mnn);
    ALLOC(idx->cut_node, (size_t)mnn + n / kCutSize + 1);   // a node's pieces: its share of the objects, rounded up
    ALLOC(idx->cut_anc, mnn);
    ALLOC(idx->cut_anc_idx, mnn);
    ALLOC(idx->node_rec, mnn);
    if (idx->metric == kAngle) ALLOC(idx->tnorm, n);
    if (idx->metric == kEdit) {
        ALLOC(idx->tstrs, (size_t)n * kStrStride);
        ALLOC(idx->tlens, n);
        ALLOC(idx->tsig, n);
        ALLOC(idx->tpack, 2 * (size_t)n);
    } else {
        ALLOC(idx->trows, (size_t)n * idx->dim);
    }
    idx->device_bytes += acct;

    BuildScratch sc;
    ALLOC(sc.node_of_pos, n);
    ALLOC(sc.ids_alt, n);
    ALLOC(sc.key, n);
    ALLOC(sc.key_alt, n);
    ALLOC(sc.split, mnn);
    ALLOC(sc.posv, n);
    ALLOC(sc.posv_alt, n);
    ALLOC(sc.lens, 3);
    ALLOC(sc.nsplit, 4);   // nodes still to split; cut nodes, their ancestors, childless nodes
    double maxnb_d = 1;   // nodes at the deepest level that can split: O^(H-2)
    for (int l = 0; l + 2 < H; l++) maxnb_d *= O;
    const bool by_segment = n <= kSegSortMax && maxnb_d <= n;
    const int maxnb = by_segment ? (int)maxnb_d : 0;
    if (by_segment) ALLOC(sc.seg, 2 * (size_t)maxnb);
#undef ALLOC
    int lid_bits = 1;
    while (lid_bits < 31 && (1 << lid_bits) < n) lid_bits++;
    size_t temp_bytes = 0, temp_lid = 0;
    GTS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, sc.key, sc.key_alt, sc.posv, sc.posv_alt, n, 0,
                                                 64, s));
    GTS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, temp_lid, (uint32_t *)nullptr, (uint32_t *)nullptr,
                                                 sc.posv_alt, sc.posv, n, 0, lid_bits, s));
    temp_bytes = std::max(temp_bytes, temp_lid);
    if (by_segment) {
        GTS_CUDA_TRY(cub::DeviceSegmentedSort::StableSortPairs(nullptr, temp_lid, sc.key, sc.key_alt, idx->id_list,
                                                               sc.ids_alt, n, maxnb, sc.seg, sc.seg, s));
        temp_bytes = std::max(temp_bytes, temp_lid);
    }
    if (dev_malloc(&sc.temp, temp_bytes ? temp_bytes : 1) != cudaSuccess) {
        cudaGetLastError();
        gts_set_error("cudaMalloc of sort scratch (%zu bytes) failed", temp_bytes);
        return GTS_ERR_NOMEM;
    }

    DevData dd{idx->dim, n, idx->metric, idx->rows, idx->strs, idx->lens};
    k_init<<<grid_for(std::max(n, mnn), 256), 256, 0, s>>>(
        n, mnn, idx->id_list, sc.node_of_pos, idx->node_pid, idx->node_size, idx->node_lid,
        idx->node_pivot, idx->node_min_dis, idx->node_flags, sc.split);
    int cur_level = 0, start = 0, split_num = 1;
    while (cur_level < H - 1 && split_num > 0) {   // tree.cuh:360
        int nb = 1;
        for (int l = 0; l < cur_level; l++) nb *= O;
        k_select_pivots<<<(nb + 255) / 256, 256, 0, s>>>(start, nb, idx->id_list, idx->node_size,
                                                         idx->node_lid, sc.split, idx->node_pivot, sc.seg);
        k_keys<<<grid_for(n, 256), 256, 0, s>>>(dd, n, start, nb, p.dis_code, p.infi_dis,
                                                 idx->id_list, sc.node_of_pos, sc.split,
                                                 idx->node_pivot, sc.key, sc.posv);
        size_t tb = temp_bytes;
        int *order = sc.posv_alt;
        if (by_segment) {
            GTS_CUDA_TRY(cudaMemcpyAsync(sc.ids_alt, idx->id_list, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, s));
            GTS_CUDA_TRY(cub::DeviceSegmentedSort::StableSortPairs(sc.temp, tb, sc.key, sc.key_alt, idx->id_list,
                                                                   sc.ids_alt, n, nb, sc.seg, sc.seg + nb, s));
        } else {
            GTS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sc.temp, tb, sc.key, sc.key_alt, sc.posv, sc.posv_alt, n, 0,
                                                         64, s));
        }
        if (!by_segment && cur_level > 0) {   // the key buffers serve the second pass
            uint32_t *lid = (uint32_t *)sc.key, *lid_alt = (uint32_t *)sc.key_alt;
            k_node_lids<<<(n + 255) / 256, 256, 0, s>>>(n, sc.posv_alt, sc.node_of_pos, idx->node_lid, lid);
            tb = temp_bytes;
            GTS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sc.temp, tb, lid, lid_alt, sc.posv_alt, sc.posv, n, 0,
                                                         lid_bits, s));
            order = sc.posv;
        }
        if (!by_segment) k_apply_order<<<(n + 255) / 256, 256, 0, s>>>(n, order, idx->id_list, sc.ids_alt);
        std::swap(idx->id_list, sc.ids_alt);
        GTS_CUDA_TRY(cudaMemsetAsync(sc.nsplit, 0, sizeof(int), s));
        long nthreads = (long)nb * O;
        k_split<<<(unsigned)((nthreads + 255) / 256), 256, 0, s>>>(
            dd, start, nb, O, p.max_size, idx->id_list, sc.split, idx->node_pid, idx->node_size,
            idx->node_lid, idx->node_pivot, idx->node_min_dis, idx->node_flags, sc.split, sc.nsplit);
        k_node_of_pos<<<grid_for(n, 256), 256, 0, s>>>(n, start, nb, O, sc.split, idx->node_size,
                                                        idx->node_lid, sc.node_of_pos);
        k_clear_level<<<(nb + 255) / 256, 256, 0, s>>>(start, nb, sc.split);
        GTS_CUDA_TRY(cudaMemcpyAsync(&split_num, sc.nsplit, sizeof(int), cudaMemcpyDeviceToHost, s));
        GTS_CUDA_TRY(cudaStreamSynchronize(s));
        GTS_CUDA_TRY(cudaGetLastError());
        start += nb;
        cur_level++;
    }
    idx->tree_h = cur_level + 1;   // tree.cuh:386
    size_t work = (size_t)n * (idx->metric == kEdit ? kStrStride : idx->dim);
    k_permute<<<grid_for(work, 256), 256, 0, s>>>(n, idx->dim, idx->metric, idx->id_list, idx->rows,
                                                  idx->trows, idx->strs, idx->tstrs, idx->lens,
                                                  idx->tlens, idx->pos_of_id);
    GTS_CUDA_TRY(cudaMemsetAsync(sc.lens, 0, 3 * sizeof(*sc.lens), s));
    if (idx->metric == kEdit) k_str_sig<<<grid_for((size_t)n, 256), 256, 0, s>>>(n, idx->tstrs, idx->tlens, idx->tsig,
                                                                             idx->tpack, sc.lens);
    if (idx->metric == kAngle) k_row_norms<<<grid_for((size_t)n, 256), 256, 0, s>>>(n, idx->dim, idx->trows, idx->tnorm);
    GTS_CUDA_TRY(cudaMemsetAsync(sc.nsplit + 1, 0, 3 * sizeof(int), s));
    k_cut_lists<<<(mnn + 255) / 256, 256, 0, s>>>(mnn, O, idx->node_flags, idx->node_size, idx->node_pivot, idx->node_lid,
                                                  idx->node_min_dis, idx->cut_node, idx->cut_anc, idx->cut_anc_idx,
                                                  sc.nsplit + 1, idx->node_rec);
    int ncuts[3] = {0, 0, 0};
    unsigned long long lens[3] = {0, 0, 0};
    GTS_CUDA_TRY(cudaMemcpyAsync(ncuts, sc.nsplit + 1, sizeof(ncuts), cudaMemcpyDeviceToHost, s));
    if (idx->metric == kEdit) GTS_CUDA_TRY(cudaMemcpyAsync(lens, sc.lens, sizeof(lens), cudaMemcpyDeviceToHost, s));
    GTS_CUDA_TRY(cudaStreamSynchronize(s));
    GTS_CUDA_TRY(cudaGetLastError());
    idx->ncut = ncuts[0];
    idx->ncut_anc = ncuts[1];
    idx->nleaf = ncuts[2];
    for (int i = 0; i < 3; i++) idx->str_lens[i] = (long long)lens[i];
    return GTS_OK;
}

int build_tree(gts_index *idx, cudaStream_t s)
{
    int rc = build_tree_impl(idx, s);
    if (rc != GTS_OK) free_tree(idx);
    return rc;
}

}  // namespace gts
