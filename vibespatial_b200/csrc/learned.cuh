// Query side of the learned cell index, shared by single joins (vs_join) and
// batch plans (vs_batch_run).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "emit.cuh"
#include "index.cuh"

namespace vs {

// Per-query scratch of the learned pipeline (points n, batch-wide cells).
struct LearnedScratch {
    void* staged = nullptr;          // striped staging regions of matched points (CellPoint)
    uint32_t* stripe_count = nullptr;
    int64_t stripe_cap = 0;
    uint32_t* cell_count = nullptr;  // counts, then start offsets after the scan
    void* grouped = nullptr;         // matched points in cell order (CellPoint)
    uint32_t* n_grouped = nullptr;
};

// Bytes of scratch for n points and n_cells cells.
size_t learned_scratch_bytes(int64_t n, int64_t n_cells);
// Carve the scratch out of one device buffer of learned_scratch_bytes().
void learned_scratch_carve(void* base, int64_t n, int64_t n_cells, LearnedScratch& sc);

// Points and jobs of one learned query; job_start is null for one job.
struct LearnedQuery {
    const double* px;
    const double* py;
    const uint8_t* pvalid;
    int64_t n;
    const LearnedJob* jobs;
    int32_t n_jobs;
    const int64_t* job_start;
    int64_t n_cells;  // batch-wide cells
    int accept_mask;
    bool sparse;         // every job's index is sparse (its occupancy bitmap is in row order)
    bool occ_rows;       // some job's index is
    bool has_ring_bins;  // some job's index has y-binned rings long enough for the split walk
    int64_t row_base;    // added to every emitted / deferred point row (chunked joins)
    LearnedShape shape;  // launch shape and ablation switches (zero = defaults)
};

// Does the map pass that queues its hits pay for an index that stores n_cells of
// its grid's grid_cells cells?  The share of points that hit is not known
// before the pass; the stored share of the grid stands for it.  10M points,
// us with and without: clustered footprints, share 0.004: 70 and 120, 0.021: 84
// and 158, 0.073: 145 and 162, 0.15: 213 and 189; points where the footprints
// are (most hit), share 0.010: 85 and 165, 0.037: 134 and 173, 0.082: 198 and
// 184; a full grid (0.90): 266 and 229.  Points that all hit and come in random
// order are the other side of this rule: 12M points, share 0.02, 428 and 387.
inline bool sparse_map_pays(int64_t n_cells, int64_t grid_cells) { return n_cells < grid_cells / 16; }
// Points from which it pays there: below, units large enough for whole lookups
// are too few to go round, and smaller ones wait for their counter.  One join
// over an index of 20k footprints (share 0.005), us with and without: 0.3M
// points 55 and 48, 1M 71 and 61, 2M 75 and 75, 2.5M 73 and 83, 5M 100 and 120,
// 12M 151 and 210; of 3k (0.0006): 1M 63 and 51, 2M 67 and 61, 2.5M 63 and 67;
// of 100k (0.02): 1M 117 and 106, 2M 135 and 132, 2.5M 134 and 143.
constexpr int64_t kSparseMapPoints = 1 << 21;

// Enqueue map -> scan -> place -> refine on stream s (no host
// synchronisation; capturable).  For one job, `single` is its descriptor
// (host copy, passed as a kernel parameter); q.jobs is used for batches.
// ctx (may be null) receives phase marks 1, 2.
int enqueue_learned(cudaStream_t s, vs_context* ctx, const LearnedQuery& q, const LearnedJob* single,
                    const LearnedScratch& sc, const PairSink& sink, const DeferSink& defer,
                    unsigned long long* counters, unsigned long long* work);

}  // namespace vs
