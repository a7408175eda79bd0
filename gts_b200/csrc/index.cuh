// index.cuh -- the gts_index handle (host side) and internal entry points.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/gts_b200.h"
#include "common.cuh"

struct gts_index {
    gts_params params;
    int num = 0, dim = 0, metric = 0;
    int tree_h = 0, max_node_num = 0;
    cudaStream_t stream = 0;

    float *rows = nullptr, *trows = nullptr;
    char *strs = nullptr, *tstrs = nullptr;
    int *lens = nullptr, *tlens = nullptr;
    uint4 *tsig = nullptr, *tpack = nullptr;   // strings in tree order: signatures, first kPackChars characters
    int *id_list = nullptr, *pos_of_id = nullptr;
    int *node_pid = nullptr, *node_size = nullptr, *node_lid = nullptr, *node_pivot = nullptr;
    float *node_min_dis = nullptr;
    uint8_t *node_flags = nullptr;
    // the batched sweep's view of the tree (sweep.cu): its cut nodes (the
    // topmost nodes of at most kCutSize objects, and larger childless ones in
    // pieces of that size) as (node, the piece's first object), their
    // ancestors with a node -> ancestor map, and for the angle metric the norms
    // of the rows in tree order
    int2 *cut_node = nullptr;
    int *cut_anc = nullptr, *cut_anc_idx = nullptr;
    int ncut = 0, ncut_anc = 0;
    int nleaf = 0;              // childless nodes with objects
    long long str_lens[3] = {}; // strings: characters, strings of more than 32 and of more than 64
    float *tnorm = nullptr;
    int4 *node_rec = nullptr;   // per node: (min_dis bits, size, first position, pivot or -1), size 0 where none exists

    // per-call scratch owned by the handle
    int *d_counter = nullptr;   // persistent-kernel work counter
    int *d_status = nullptr;    // kernel status word
    unsigned long long *d_stats = nullptr;   // work counters of the last search (kStatsN)
    bool keep_stats = false;                 // a nested search adds to, not resets, the counters
    size_t device_bytes = 0;

    // tensor-core filter (L2): per-block operand records, built on first use
    unsigned char *fast_recs = nullptr;
    int fast_nb = 0, fast_nsb = 0;   // filter blocks, superblocks
    int last_fast_overflow = 0;
    // device time of the filter kernel (CUDA events around each launch),
    // kept only while timing is on (gts_filter_timing)
    bool time_filter = false;
    cudaEvent_t fev[2] = {nullptr, nullptr};
    double filter_ms = 0.0;
    long long filter_launches = 0;
    // kernels this library launched for searches on this handle (host count)
    long long kernel_launches = 0;
    // autotuned fast-form configuration per k (fast.cu): 0 = not tuned, else
    // 1 | learned << 1 | column groups << 2 | blocks per item << 8
    int fast_cfg[65] = {};
    int range_variant = 1;   // fast range counts: 0 the block-stationary filter where it fits, 1 the tile filter
    // autotuned threads per query CTA of the plain traversal per search mode
    // (kNN, range count, range ids; search.cu), 0 = not tuned
    static constexpr int kSplitDefault = 32768;
    int plain_nt[3] = {};
    // its query CTAs of 128 / 256 / 512 threads resident at once (0: not asked yet)
    int cta_resident[3] = {};
    // set by a caller: pinned threads or a hand-over threshold choose the
    // traversal over the batched sweep
    bool plain_pinned[3] = {};
    bool plain_split_set = false;
    // batches large enough to tune went to another search: no threads chosen yet
    bool plain_passed[3] = {};
    // range counts: objects a query verifies in one CTA before it hands its
    // older stack entries over as (query, node) items (0: never); the item
    // lists, and the items handed over since the last reset
    int plain_split = kSplitDefault;
    void *split_buf = nullptr;
    size_t split_bytes = 0;
    long long last_split_items = 0;

    // reusable per-call scratch (grown on demand, freed with the handle)
    void *scratch = nullptr;
    size_t scratch_bytes = 0;
    // device copies of host-buffer arguments (gts_knn, gts_range, ...):
    // grown on demand and kept, so those calls allocate nothing in steady state
    void *io = nullptr;
    size_t io_bytes = 0;
    // the fast form's small batches (fast_small.cu): lists, and a result word
    // in host memory; pinned configurations keep a k on the tiles
    void *small_buf = nullptr;
    size_t small_bytes = 0;
    int *small_result = nullptr;
    bool fast_pinned[65] = {};
    // hits of a range-ids run on their way to the host
    void *hits = nullptr;
    size_t hits_bytes = 0;
    // scratch of the running call outside `scratch` (search_budget)
    size_t held_bytes = 0;
    // CUDA graph of the fast form's filter pass (fast.cu), launched on the
    // handle's own stream and replayed while the batch shape stays the same
    cudaStream_t graph_stream = nullptr;
    // up to kGraphSlots captured filter passes, one per batch shape and
    // argument buffers (batches of a few shapes in turn, such as one per k,
    // each replay their own), least recently used replaced
    static constexpr int kGraphSlots = 16;
    cudaGraphExec_t graph_exec[kGraphSlots] = {};
    long long graph_key[kGraphSlots][8] = {};
    long long graph_used[kGraphSlots] = {};
    long long graph_kernels[kGraphSlots] = {};   // this library's kernels in each graph
    cudaEvent_t graph_ev[2] = {nullptr, nullptr};
    bool use_graphs = true;
    long long graph_launches = 0;
    long long graph_clock = 0;

    // learned kNN radius (mlp.cu): parameters, input standardisation,
    // feature pivots; valid for the tree it was trained on
    float *mlp_P = nullptr, *mlp_norm = nullptr;
    int *mlp_piv = nullptr;
    int mlp_npiv = 0;
    float mlp_ymu = 0.f, mlp_ysig = 1.f, mlp_widen = 1.f;
    float mlp_widen_at[65] = {};   // per trained k (0: none; the global factor serves)
    bool mlp_ready = false;

    gts::DevTree dev() const;
};

namespace gts {

// Search work counters (gts_search_stats):
//   [0] plain: leaf objects read          fast: operand blocks streamed
//   [1] plain: pivots evaluated           fast: bytes streamed
//   [2] exact (reference-order) values    [3] plain: queries finished
//   [4] fast: queries answered again on the plain path
//   [5] fast: candidates appended         [6] fast: filter passes
//   [7] fast: (query tile, block) pairs tested by the block bound
constexpr int kStatsN = 8;
constexpr int kPackChars = 32;
constexpr int kCutSize = 128;   // objects of a cut node (or a piece of one) at most

// Build the tree for the data already placed in idx->rows / strs / lens.
int build_tree(gts_index *idx, cudaStream_t s);
// Free the tree arrays (not the data).
void free_tree(gts_index *idx);
void free_data(gts_index *idx);

int search_knn(gts_index *idx, const int *d_qids, int qnum, int k, int form,
               float *d_kth, int *d_ids, float *d_dists, cudaStream_t s);
int search_range(gts_index *idx, const int *d_qids, int qnum, float r, int *d_counts,
                 const uint32_t *d_deleted, cudaStream_t s);
int search_range_fast(gts_index *idx, const int *d_qids, int qnum, float r, int *d_counts, cudaStream_t s);
// Range counts at time stamps (the stream-update path): query q is object
// d_qids[q] at operation d_qtime[q]; an object within r adds its entries
// live in the tree (d_tree_counts) and in the cache list (d_cache_counts)
// at that operation (SearchArgs::ents).
int search_range_timed(gts_index *idx, const int *d_qids, const int *d_qtime, int qnum, float r,
                       const int *d_ent_off, const int4 *d_ents, int *d_tree_counts, int *d_cache_counts,
                       cudaStream_t s);
// Queries given as data (rows, or strings with lengths), not ids: no self
// match; the plain traversal.
int search_knn_rows(gts_index *idx, const float *d_qrows, const char *d_qstrs, const int *d_qlens, int qnum, int k,
                    float *d_kth, int *d_ids, float *d_dists, cudaStream_t s);
int search_range_rows(gts_index *idx, const float *d_qrows, const char *d_qstrs, const int *d_qlens, int qnum,
                      float r, int *d_counts, cudaStream_t s);
int search_range_ids(gts_index *idx, const int *d_qids, int qnum, float r, int *d_counts,
                     int *d_ids, float *d_dists, const int *d_offsets, cudaStream_t s);
// Range counts and hits in one pass over the data (host outputs; hits only
// up to `capacity`), ordered by (distance, id) per query.  *done = 0: not a
// batch the sweep answers in full; *total: hits of all queries.
int sweep_range_ids(gts_index *idx, const int *d_qids, int qnum, float r, int *d_counts, int *counts_out,
                    int *offsets_out, int *ids_out, float *dists_out, size_t capacity, size_t *total, int *done,
                    cudaStream_t s);

// Device memory (memory.cu): as cudaMalloc / cudaFree, with freed blocks of
// 64 KiB and more kept for the next request, up to a bound.
cudaError_t dev_malloc(void **p, size_t bytes);
void dev_free(void *p);

template <typename T>
int dev_alloc(T **p, size_t n, size_t *acct);

// Device scratch one search call may hold (gts_params.mem_budget_gb; 0 means
// 8 GiB), less what the call holds already around a search of its own.  The
// fast form and the sweeps size their runs of queries, the seeded plain form
// its chunks and the update path its query batches to fit it.
inline size_t search_budget(const gts_index *idx)
{
    const double gb = idx->params.mem_budget_gb;
    const size_t b = gb > 0 ? (size_t)(gb * 1073741824.0) : ((size_t)8 << 30);
    return b > idx->held_bytes ? b - idx->held_bytes : 0;
}

// Grow idx->scratch to at least `bytes`.
int ensure_scratch(gts_index *idx, size_t bytes);
// Grow idx->io to at least `bytes`.
int ensure_io(gts_index *idx, size_t bytes);
// idx->hits of at least `bytes`, at most `room` where it grows.
int ensure_hits(gts_index *idx, size_t bytes, size_t room, void **out);

bool fast_supported(const gts_index *idx, int k);
int mlp_seed(gts_index *idx, const int *d_qids, int qnum, int k, int *d_r2_bits, cudaStream_t st);
int search_knn_fast(gts_index *idx, const int *d_qids, int qnum, int k, float *d_kth, int *d_ids,
                    float *d_dists, cudaStream_t s);
int search_knn_plain_learned(gts_index *idx, const int *d_qids, int qnum, int k, float *d_kth, int *d_ids,
                             float *d_dists, cudaStream_t s);
int fast_config_get(const gts_index *idx, int k, int *tuned, int *learned, int *cg, int *item, int *variant);
int fast_prepare_now(gts_index *idx, cudaStream_t st, int *done);
// Drop the captured filter graph (its device pointers or parameters changed).
void graph_invalidate(gts_index *idx);
// Unseeded filter with all scratch inside the caller's fixed buffer.
int search_knn_fast_fixed(gts_index *idx, const int *d_qids, int qnum, int k, float *d_kth, int *d_ids,
                          float *d_dists, unsigned char *scratch, size_t bytes, cudaStream_t s);

// A set of device allocations freed together on scope exit.
struct DevVec {
    void *ps[8] = {};
    int n = 0;
    ~DevVec()
    {
        for (int i = 0; i < n; i++)
            if (ps[i]) dev_free(ps[i]);
    }
    template <typename T>
    int alloc(T **p, size_t cnt)
    {
        int rc = dev_alloc(p, cnt, nullptr);
        if (rc == 0 && n < 8) ps[n++] = *p;
        return rc;
    }
};

}  // namespace gts
