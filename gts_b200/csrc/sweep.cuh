// sweep.cuh -- what the row sweep (sweep.cu) and the string sweep
// (sweep_edit.cu) share.
#pragma once
#include "search.cuh"

namespace gts {

struct SweepArgs {
    SearchArgs a;
    int q0, nq, ntiles, Qp, ld;         // the run's queries a.qids[q0 ..], padded count, query row stride
    int tq;                             // queries per tile (row lists, ring bounds)
    int ncut, nanc;
    const int *cut, *anc, *anc_idx;
    const float *tnorm;                 // angle: norms of the rows in tree order
    int *key, *order;                   // tree position of the query; sorted order -> query of the run
    int *bq;                            // sorted slot -> query of the batch (-1: padding)
    float *seed;                        // per query of the run: bound on the k-th distance (kNN)
    float *qrow;                        // [Qp][ld] sorted query rows, zero padded
    float *R, *vthr, *vlow, *qnorm;     // per sorted query: radius, value thresholds
    int *self;                          // its tree position when it is an object (-1)
    float *dlo, *dhi;                   // [nanc][Qp] pivot distance bounds
    int *nrows, *rowpos;                // per tile: rows to look at, their positions [ntiles][num]
    int *ccnt, *cpos;                   // candidate lists [Qp][cap]
    float *cv;
    int *cnt, *cnt2;                    // range: certain counts per sorted query
    int *ctr;                           // [0] item counter, [1] queries left over
    int4 *left;                         // queries whose list overflowed: (query, 0, 0, 0) for the traversal
    float *left_R;                      // kNN: and a bound on their k-th distance, from the list
    const int4 *again;                  // kNN, a later round: the run's queries and bounds come from
    const float *again_R;               //   again[q0 ..], again_R[q0 ..]
    int cap;                            // candidates listed per query
    int sample;                         // look at every sample-th row only (1: all)
    const uint4 *lens_ok;               // strings: per tile a mask of the lengths some query can match (nullable)
};

// Ring bounds: the rows of the cut nodes that some query of each tile can
// reach, appended to the tiles' row lists (nrows zeroed by the caller).
void sweep_cut_launch(const SweepArgs &s, int ntiles, cudaStream_t st);

// The string sweep (edit distance); as run_sweep.
int run_sweep_edit(gts_index *idx, const SearchArgs &a, cudaStream_t st, int *done, const int4 **items, int *n_left);

}  // namespace gts
