// Host-side launchers shared by the C-ABI translation unit.
#pragma once
#include <stdint.h>

#include "emit.cuh"
#include "index.cuh"
#include "primitives.cuh"
#include "vs_common.cuh"

namespace vs {
// Query points keyed by their level-16 Hilbert key in the polygon frame and
// radix-sorted; order[0, *n_valid) are the points that can match.
struct QueryOrder {
    Scratch<uint32_t> keys, order, n_valid;
};
// clamp: keep points outside the polygon frame (keyed at the frame's edge),
// as distance joins need them; otherwise they are left out.
int prepare_queries(vs_context* ctx, const vs_index* idx, const vs_points* pts, QueryOrder& q, bool clamp = false);
int accept_mask_for(int predicate, int* mask);
// row_base is added to every emitted or deferred point row (a chunk of a
// larger point array); the exact pass subtracts it to read the chunk's points.
int launch_rtree_join(vs_context* ctx, const vs_index* idx, const vs_points* pts, int accept_mask, bool brute,
                      bool bulk_leaves, int32_t* d_left, int32_t* d_right, int64_t capacity, const DeferSink& dsink,
                      int64_t row_base = 0);
// Whether a learned join of n points runs as one direct launch (no grouping):
// while the records it tests, n times the mean list length of a cell, stay
// below kDirectWork.  Whole sorted calls, direct against grouped, us:
//   1000 stars (lists of 2.5)     32k 114/189  262k 158/217  1M 280/309
//   50k stars (30)                1k 126/488   32k 354/547   65k 607/589
//   100k footprints, UTM (1.2)    32k 35/165   262k 109/180  1M 145/204
//   1M footprints, Zipf (2.4)     32k 108/235  524k 235/297  1M 336/336
//   40k with holes, parts (12)    8k 149/255   131k 290/302  262k 444/360
constexpr int64_t kDirectPoints = 1 << 20;
constexpr double kDirectWork = 1.5e6;
inline bool direct_join_pays(const vs_index* idx, int64_t n) {
    return n <= kDirectPoints && (double)n * idx->learned.mean_list <= kDirectWork;
}
// Enqueue it; after the stream has been waited for, ctx->h_counter holds the
// kDirect* words (ticket: whether the pairs are sorted, start: device time in ns).
int launch_direct_join(vs_context* ctx, const vs_index* idx, const vs_points* pts, int accept_mask, int32_t* d_left,
                       int32_t* d_right, int64_t capacity, bool sort);
int launch_learned_join(vs_context* ctx, const vs_index* idx, const vs_points* pts, int accept_mask,
                        int32_t* d_left, int32_t* d_right, int64_t capacity, const DeferSink& dsink,
                        int64_t row_base = 0, const LearnedShape& shape = LearnedShape{});
// Exact pass over the pairs the filtered kernels deferred (count read on device).
int launch_resolve_deferred(vs_context* ctx, const vs_index* idx, const vs_points* pts, int accept_mask,
                            int32_t* d_left, int32_t* d_right, int64_t capacity, const DeferSink& dsink,
                            int64_t row_base = 0);
// Grow the context's deferred-pair buffer to at least `want` pairs.
int ensure_defer_capacity(vs_context* ctx, unsigned long long want);
// Release the context's vs_join_host pipeline (streams, events, buffers).
void free_host_pipe(vs_context* ctx);
int launch_locate_aligned(vs_context* ctx, const vs_points* pts, const vs_polygons* polys, uint8_t* d_out);
// Sort (left, right) pairs and wait for them; rows below max_left, max_right.
int sort_pairs(vs_context* ctx, int32_t* d_left, int32_t* d_right, int64_t n, uint64_t max_left,
               uint64_t max_right);
// The same without waiting (by_runs as for radix_sort_pairs, on
// d_counters[kStatus], which clear_status zeroes).
int enqueue_sort_pairs(vs_context* ctx, int32_t* d_left, int32_t* d_right, int64_t n, uint64_t max_left,
                       uint64_t max_right, bool by_runs);
// Wait for an enqueued sort (by_runs), and sort by every digit what it left
// (`sorted`, an event behind the first sort, is then recorded again).
int finish_sort_pairs(vs_context* ctx, int32_t* d_left, int32_t* d_right, int64_t n, uint64_t max_left,
                      uint64_t max_right, cudaEvent_t sorted = nullptr);
// Zero the status word; wait for the stream and read it (to the last word of
// h_counter; VS_E_TIMEOUT for a wait that gave up).
int clear_status(vs_context* ctx);
int finish_status(vs_context* ctx);
int build_rtree(vs_context* ctx, const vs_polygons* P, vs_index* idx);
// y-bins for rings of at least min_vertices vertices (0: the default, < 0: none).
int build_ring_bins(vs_context* ctx, vs_index* idx, int min_vertices);
void free_index_memory(vs_index* idx);
int hilbert_point_keys(const double* x, const double* y, int64_t n, double minx, double miny, double maxx,
                       double maxy, uint64_t* keys, cudaStream_t s);
}  // namespace vs
