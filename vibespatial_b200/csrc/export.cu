// Join export on the device: the row indexers of a relation join for
// how = inner / left / right / outer, after on_attribute filtering.
//
// Replaces the reference's host export (src/vibespatial/api/_native_results.py:395-470,
// _adjust_join_indexers) and its shared-attribute filter
// (src/vibespatial/api/tools/sjoin.py:826-888, filter_by_equal_columns).
// Input pairs are sorted by (left, right), as every join here returns them.
//
//   1. attribute filter (equal codes, missing codes never match): one pass
//      that compacts the kept pairs and their source positions in order
//   2. how = right: the kept pairs re-sorted by (right, left) (radix sort)
//   3. one read of the driving rows (left rows; right rows for how = right)
//      finds each tile of 2048 rows' first pair and its matched rows, which a
//      scan sums; a tile's output is one contiguous range, which one block
//      writes in order (a row's pairs, or one row with -1 on the other side
//      when it has none)
//   4. how = outer: right rows no pair reaches are appended in order
// The sizes stay on the device until the end: the writing kernels check them
// (rows out of range, output capacity) themselves, and one wait returns them.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "join.cuh"
#include "primitives.cuh"
#include "vs_common.cuh"

namespace vs {
namespace {

// Device-side sizes and flags of one export.
struct ExportState {
    uint32_t bad;         // pairs naming rows out of range
    uint32_t unsorted;    // pairs whose driving row is below the one before
    uint32_t kept;        // pairs after the filter
    uint32_t appended;    // how = outer: right rows without a pair
    uint32_t distinct;    // driving rows with a pair
    uint32_t ticket;
    uint32_t timeout;
    uint32_t pad;
};

// Without a filter every pair is kept; those whose rows fall outside
// [0, n_left) x [0, n_right) are counted.
__global__ void export_check_kernel(const int32_t* __restrict__ l, const int32_t* __restrict__ r, int64_t n,
                                    int64_t n_left, int64_t n_right, ExportState* __restrict__ st) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->kept = (uint32_t)n;
    uint32_t b = 0;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        b += (l[k] < 0 || l[k] >= n_left || r[k] < 0 || r[k] >= n_right) ? 1u : 0u;
    if (b) atomicAdd(&st->bad, b);
}

constexpr int kFilterThreads = 256;
constexpr int kFilterItems = 8;
constexpr int kFilterTile = kFilterThreads * kFilterItems;
constexpr int kFilterWait = 1 << 20;  // polls of earlier tiles before a tile gives up

// The attribute filter in one pass: a tile's kept pairs (equal codes, rows in
// range; others are counted as bad) go to the place that the tiles before it
// leave (look-back over their counts, value << 2 | 1, then sums, value << 2 |
// 2, 32 at a time; tiles are taken in order, so those before are running or
// done).  8.6M pairs of 20M x 400k rows: keep flags, their scan and the
// compaction took 153 us.
__global__ void __launch_bounds__(kFilterThreads) export_filter_kernel(
    const int32_t* __restrict__ l, const int32_t* __restrict__ r, int64_t n, int64_t n_left, int64_t n_right,
    const int64_t* __restrict__ lc, const int64_t* __restrict__ rc, int32_t* __restrict__ ol, int32_t* __restrict__ orr,
    uint32_t* __restrict__ osrc, unsigned long long* tiles, ExportState* st) {
    __shared__ uint32_t s_tile, s_bad;
    __shared__ uint32_t s_w[kFilterThreads / 32];
    __shared__ uint32_t s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_tile = atomicAdd(&st->ticket, 1u);
        s_bad = 0;
    }
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t base = tile * kFilterTile + (int64_t)warp * 32 * kFilterItems + lane;
    // a warp's items lie together, 32 a round: its kept pairs stay in order
    int32_t li[kFilterItems], ri[kFilterItems];
    uint32_t keep = 0, bad = 0, mine = 0;
    uint32_t before[kFilterItems];
#pragma unroll
    for (int u = 0; u < kFilterItems; ++u) {
        const int64_t k = base + u * 32;
        li[u] = ri[u] = -1;
        if (k < n) {
            li[u] = l[k];
            ri[u] = r[k];
        }
    }
    int64_t a[kFilterItems], c[kFilterItems];
#pragma unroll
    for (int u = 0; u < kFilterItems; ++u) {
        const bool ok = li[u] >= 0 && li[u] < n_left && ri[u] >= 0 && ri[u] < n_right;
        bad += !ok && base + u * 32 < n ? 1u : 0u;
        a[u] = ok ? lc[li[u]] : -1;
        c[u] = ok ? rc[ri[u]] : -2;
    }
#pragma unroll
    for (int u = 0; u < kFilterItems; ++u) {
        const bool kp = a[u] >= 0 && a[u] == c[u];
        const unsigned m = __ballot_sync(0xffffffffu, kp);
        before[u] = mine + __popc(m & ((1u << lane) - 1u));
        mine += __popc(m);  // warp-uniform
        keep |= kp ? 1u << u : 0u;
    }
    if (lane == 0) s_w[warp] = mine;
    if (bad) atomicAdd(&s_bad, bad);
    __syncthreads();
    if (warp == 0) {
        uint32_t total = 0;
        for (int w = 0; w < kFilterThreads / 32; ++w) total += s_w[w];
        if (lane == 0 && tile > 0) atomicExch(&tiles[tile], ((unsigned long long)total << 2) | 1ull);
        unsigned long long sum = 0;
        int polls = 0;
        for (int64_t t = tile - 1; t >= 0;) {
            unsigned long long w = 2ull;  // before the first tile: a sum of 0
            if (t - lane >= 0) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(&tiles[t - lane]) : "memory");
            const unsigned sums = __ballot_sync(0xffffffffu, (w & 3) == 2);
            const unsigned missing = __ballot_sync(0xffffffffu, (w & 3) == 0);
            const int stop = sums ? __ffs(sums) - 1 : 32;   // nearest tile with a sum
            const int gap = missing ? __ffs(missing) - 1 : 32;
            const int take = stop < gap ? stop + 1 : gap;   // lanes whose values count
            unsigned long long v = lane < take ? w >> 2 : 0ull;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            sum += v;
            if (stop < gap) break;
            t -= take;
            if (take == 0 && ++polls > kFilterWait) {
                if (lane == 0) atomicOr(&st->timeout, 1u);
                break;
            }
        }
        if (lane == 0) {
            atomicExch(&tiles[tile], ((sum + total) << 2) | 2ull);
            s_base = (uint32_t)sum;
            if ((tile + 1) * kFilterTile >= n) st->kept = (uint32_t)(sum + total);
            if (s_bad) atomicAdd(&st->bad, s_bad);
        }
    }
    __syncthreads();
    uint32_t pos0 = s_base;
    for (int w = 0; w < warp; ++w) pos0 += s_w[w];
#pragma unroll
    for (int u = 0; u < kFilterItems; ++u) {
        if (!((keep >> u) & 1u)) continue;
        const int64_t p = (int64_t)pos0 + before[u];
        if (p >= n) continue;  // only after a wait that gave up
        ol[p] = li[u];
        orr[p] = ri[u];
        osrc[p] = (uint32_t)(base + u * 32);
    }
}

// (driving row, other row) keys; vals = position in the kept pairs
__global__ void export_keys_kernel(const int32_t* __restrict__ drive, const int32_t* __restrict__ other, int64_t n,
                                   uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        keys[k] = ((uint64_t)(uint32_t)drive[k] << 32) | (uint32_t)other[k];
        vals[k] = (uint32_t)k;
    }
}

// The kept pairs in driving order: as they are, or through sorted keys.
struct ExportPairs {
    const int32_t* l;        // driving rows (null: keys)
    const int32_t* o;        // other rows
    const uint64_t* keys;    // driving row << 32 | other row, sorted
    const uint32_t* perm;    // with keys: position in the kept pairs
    const uint32_t* src;     // source position of a kept pair (null: its own)
    __device__ __forceinline__ int32_t drive(int64_t k) const { return l ? l[k] : (int32_t)(keys[k] >> 32); }
    __device__ __forceinline__ int32_t other(int64_t k) const { return l ? o[k] : (int32_t)(keys[k] & 0xffffffffull); }
    __device__ __forceinline__ int64_t source(int64_t k) const {
        const uint32_t j = l ? (uint32_t)k : perm[k];
        return src ? (int64_t)src[j] : (int64_t)j;
    }
};

constexpr int kTileThreads = 256;
constexpr int kTileRows = 2048;
constexpr int kRowsPerThread = kTileRows / kTileThreads;

// Of every tile of driving rows: its first pair (first[n_tiles] = the pairs)
// and how many of its rows have one.  A pair that begins a row fills the tiles
// from the row before: n_tiles stores in all while the rows ascend.  Pairs that
// do not are found in the same read, and the stores, whose result is thrown
// away then, end at the next look at that flag: shuffled pairs would fill
// n_tiles / 3 for every ascent (2M pairs over 20M rows: 77 ms).  A search for
// every tile's first pair is bounded too, but took 4 us more for sorted pairs.
__global__ void export_bounds_kernel(const ExportPairs pairs, int64_t n_drive, int64_t n_tiles,
                                     uint32_t* __restrict__ first, uint32_t* __restrict__ matched, ExportState* st) {
    const int64_t m = st->kept;
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~(int64_t)31; b < m; b += stride) {
        const int64_t k = b + lane;
        int32_t row = -1, prev = -1;
        if (k < m) {
            row = pairs.drive(k);
            prev = k > 0 ? pairs.drive(k - 1) : -1;
        }
        const bool ok = k < m && row >= 0 && row < n_drive && prev >= -1 && prev < n_drive;  // (else counted as bad)
        if (ok && row < prev) st->unsorted = 1u;
        const bool fresh = ok && row > prev;
        const int64_t tile = ok ? row / kTileRows : -1;
        if (fresh) {
            const int64_t from = prev < 0 ? 0 : prev / kTileRows + 1;
            for (int64_t t = from; t <= tile; ++t) {
                first[t] = (uint32_t)k;
                if (((t - from) & 31) == 31 && *(volatile uint32_t*)&st->unsorted) break;
            }
        }
        if (ok && k == m - 1)
            for (int64_t t = tile + 1; t <= n_tiles; ++t) first[t] = (uint32_t)m;
        // a warp's rows mostly lie in one tile
        const int64_t t0 = __shfl_sync(0xffffffffu, tile, 0);
        const unsigned same = __ballot_sync(0xffffffffu, fresh && tile == t0);
        if (lane == 0 && same) atomicAdd(&matched[t0], (uint32_t)__popc(same));
        if (fresh && tile != t0) atomicAdd(&matched[tile], 1u);
    }
}

__device__ __forceinline__ bool export_writes(const ExportState* st, int64_t n_drive, int64_t capacity) {
    return st->bad == 0 && st->unsorted == 0 && st->timeout == 0 &&
           (int64_t)st->kept + (n_drive - (int64_t)st->distinct) + (int64_t)st->appended <= capacity;
}

// A driving row's share of the output, packed: its pairs in the low word,
// 1 in the high word when it has none (it then owns one unmatched row).
// Neither word carries into the other: pairs and rows are below 2^31.
__device__ __forceinline__ uint64_t row_pack(uint32_t c) { return (uint64_t)c | ((uint64_t)(c == 0u) << 32); }

// One block per tile of driving rows.  The tile's pairs are the run
// [first[tile], first[tile + 1]), counted per row in shared memory; its output
// starts at its pairs before it plus the unmatched rows before it.  Row k of
// the tile owns [s_start[k], s_start[k + 1]) of it and its pairs are
// [s_first[k], s_first[k + 1]) of the tile's pairs.  Output positions go to
// consecutive threads, so the stores are contiguous; the owner of a position
// is marked in shared memory (searched for in tiles with more outputs).
// Bound by the 24 bytes a row it writes.  21M rows: 165 us with per-row counts
// read from memory and a search for every output row.
// Tiles of many pairs take several blocks (gridDim.y), each of which counts
// the tile's pairs and writes its share of the output: 1000 rows of 400 pairs,
// one tile, are a call of 1328 us with one block and of 201 with 24.
constexpr int kOwners = 4096;
constexpr int64_t kBlockPairs = 16384;  // pairs a tile has on average for each of its blocks, at most kTileBlocks
constexpr int kTileBlocks = 64;

__global__ void __launch_bounds__(kTileThreads) export_write_kernel(
    const ExportPairs pairs, int64_t n_drive, const uint32_t* __restrict__ first, const uint32_t* __restrict__ matched,
    const ExportState* __restrict__ st, int64_t capacity, int64_t* __restrict__ o_drive, int64_t* __restrict__ o_other,
    int64_t* __restrict__ o_src) {
    __shared__ uint32_t s_start[kTileRows + 1];
    __shared__ uint32_t s_first[kTileRows + 1];  // first the rows' counts
    __shared__ uint16_t s_owner[kOwners];
    __shared__ uint64_t s_w[kTileThreads / 32];
    if (!export_writes(st, n_drive, capacity)) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int64_t base = (int64_t)blockIdx.x * kTileRows;
    const int64_t p0 = first[blockIdx.x], p1 = first[blockIdx.x + 1];
    for (int k = t; k < kTileRows; k += kTileThreads) s_first[k] = 0;
    __syncthreads();
    for (int64_t k = p0 + t; k < p1; k += kTileThreads) atomicAdd(&s_first[pairs.drive(k) - base], 1u);
    __syncthreads();
    uint64_t v[kRowsPerThread];
    uint64_t sum = 0;
#pragma unroll
    for (int k = 0; k < kRowsPerThread; ++k) {
        const int row = t * kRowsPerThread + k;
        v[k] = base + row < n_drive ? row_pack(s_first[row]) : 0ull;  // rows past the end own nothing
        sum += v[k];
    }
    uint64_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    uint64_t run = incl - sum;
    for (int w = 0; w < warp; ++w) run += s_w[w];
#pragma unroll
    for (int k = 0; k < kRowsPerThread; ++k) {
        s_first[t * kRowsPerThread + k] = (uint32_t)run;
        const uint32_t at = (uint32_t)run + (uint32_t)(run >> 32);
        s_start[t * kRowsPerThread + k] = at;
        const uint32_t owned = (uint32_t)v[k] + (uint32_t)(v[k] >> 32);
        for (uint32_t o = at; o < at + owned && o < (uint32_t)kOwners; ++o) s_owner[o] = (uint16_t)(t * kRowsPerThread + k);
        run += v[k];
    }
    if (t == kTileThreads - 1) {
        s_first[kTileRows] = (uint32_t)run;
        s_start[kTileRows] = (uint32_t)run + (uint32_t)(run >> 32);
    }
    __syncthreads();
    const int64_t out_base = p0 + (base - (int64_t)matched[blockIdx.x]);
    const uint32_t total = s_start[kTileRows];
    for (uint32_t o = blockIdx.y * kTileThreads + t; o < total; o += gridDim.y * kTileThreads) {
        // the row that owns o: s_start[lo] <= o < s_start[lo + 1]
        int lo = 0;
        if (o < (uint32_t)kOwners) {
            lo = s_owner[o];
        } else {
            int hi = kTileRows;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (s_start[mid] <= o) lo = mid;
                else hi = mid;
            }
        }
        const uint32_t f0 = s_first[lo];
        const int64_t p = out_base + o;
        o_drive[p] = base + lo;
        if (s_first[lo + 1] == f0) {
            o_other[p] = -1;
            if (o_src) o_src[p] = -1;
        } else {
            const int64_t k = p0 + f0 + (o - s_start[lo]);
            o_other[p] = pairs.other(k);
            if (o_src) o_src[p] = pairs.source(k);
        }
    }
}

__global__ void export_mark_kernel(const int32_t* __restrict__ r, int64_t n_right, uint32_t* __restrict__ matched,
                                   const ExportState* __restrict__ st) {
    const int64_t n = st->kept;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        if (r[k] >= 0 && r[k] < n_right) matched[r[k]] = 1u;  // (others are counted as bad)
}

__global__ void export_flip_kernel(uint32_t* __restrict__ v, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[i] = v[i] ? 0u : 1u;
}

__global__ void export_append_kernel(const uint32_t* __restrict__ missing, const uint32_t* __restrict__ pos,
                                     int64_t n, const ExportState* __restrict__ st, int64_t n_drive, int64_t capacity,
                                     int64_t* __restrict__ o_left, int64_t* __restrict__ o_right,
                                     int64_t* __restrict__ o_src) {
    if (!export_writes(st, n_drive, capacity)) return;
    const int64_t base = (int64_t)st->kept + (n_drive - (int64_t)st->distinct);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (missing[i]) {
            const int64_t p = base + pos[i];
            o_left[p] = -1;
            o_right[p] = i;
            if (o_src) o_src[p] = -1;
        }
}

__global__ void export_copy_kernel(const int32_t* __restrict__ l, const int32_t* __restrict__ r,
                                   const uint32_t* __restrict__ src, const ExportState* __restrict__ st,
                                   int64_t capacity, int64_t* __restrict__ ol, int64_t* __restrict__ orr,
                                   int64_t* __restrict__ osrc) {
    const int64_t n = st->kept;
    if (st->bad || st->timeout || n > capacity) return;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        ol[k] = l[k];
        orr[k] = r[k];
        if (osrc) osrc[k] = src ? (int64_t)src[k] : k;
    }
}

template <class K>
int grid_of(K kernel, int64_t n) {
    return resident_grid(kernel, n > 0 ? n : 1, 256);
}

}  // namespace
}  // namespace vs

using namespace vs;

extern "C" {

int vs_join_export(vs_context* ctx, const int32_t* d_left, const int32_t* d_right, int64_t n_pairs, int64_t n_left,
                   int64_t n_right, int32_t how, const int64_t* d_left_code, const int64_t* d_right_code,
                   int64_t* d_out_left, int64_t* d_out_right, int64_t* d_out_src, int64_t capacity,
                   int64_t* n_out) {
    if (!ctx || !n_out || (n_pairs > 0 && (!d_left || !d_right))) {
        set_error("ctx/n_out/pairs is NULL");
        return VS_E_ARG;
    }
    *n_out = 0;
    if (how < VS_HOW_INNER || how > VS_HOW_OUTER) {
        set_error("unknown how code %d", how);
        return VS_E_ARG;
    }
    if (n_pairs < 0 || n_pairs > 0x7fffffffLL || n_left < 0 || n_left > 0x7fffffffLL || n_right < 0 ||
        n_right > 0x7fffffffLL) {
        set_error("sizes outside the 32-bit ranges (pairs %lld, left %lld, right %lld)", (long long)n_pairs,
                  (long long)n_left, (long long)n_right);
        return VS_E_ARG;
    }
    // codes for one side imply codes for the other (an empty side may pass NULL)
    const bool with_codes = d_left_code || d_right_code;
    if (with_codes && ((n_left > 0 && !d_left_code) || (n_right > 0 && !d_right_code))) {
        set_error("attribute codes must be given for both sides or neither");
        return VS_E_ARG;
    }
    if (capacity < 0 || (capacity > 0 && (!d_out_left || !d_out_right))) {
        set_error("invalid output buffers (capacity %lld)", (long long)capacity);
        return VS_E_ARG;
    }
    VS_TRY(use_device(ctx->device));
    cudaStream_t s = ctx->stream;
    Scratch<ExportState> state;
    VS_TRY(state.alloc(1, s));
    ExportState h{};
    VS_CUDA_TRY(cudaMemsetAsync(state.p, 0, sizeof(h), s));
    // the state after all passes so far, and what it says of the pairs
    auto read_state = [&]() -> int {
        VS_CUDA_TRY(cudaMemcpyAsync(&h, state.p, sizeof(h), cudaMemcpyDeviceToHost, s));
        VS_CUDA_TRY(cudaStreamSynchronize(s));
        if (h.bad) {
            set_error("%u pairs name rows outside [0, %lld) x [0, %lld)", h.bad, (long long)n_left, (long long)n_right);
            return VS_E_ARG;
        }
        if (h.timeout) {
            set_error("a bounded device wait (export filter) gave up");
            return VS_E_TIMEOUT;
        }
        return VS_OK;
    };
    auto over_capacity = [&](int64_t rows) {
        *n_out = rows;
        if (rows <= capacity) return VS_OK;
        set_error("output holds %lld rows, %lld required", (long long)capacity, (long long)rows);
        return VS_E_CAPACITY;
    };
    // 1. attribute filter (ordered compaction); without codes the pairs are used in place
    const int32_t* kl = d_left;
    const int32_t* kr = d_right;
    const uint32_t* ksrc = nullptr;  // null: position k is its own source
    Scratch<uint32_t> ksrc_buf;
    Scratch<int32_t> kl_buf, kr_buf;
    Scratch<unsigned long long> filter_tiles;
    if (n_pairs > 0 && !with_codes) {
        export_check_kernel<<<grid_of(export_check_kernel, n_pairs), 256, 0, s>>>(d_left, d_right, n_pairs, n_left,
                                                                                  n_right, state.p);
        VS_LAUNCHED("export_check", s);
    }
    if (with_codes && n_pairs > 0) {
        const int64_t tiles = (n_pairs + kFilterTile - 1) / kFilterTile;
        VS_TRY(kl_buf.alloc((size_t)n_pairs, s));
        VS_TRY(kr_buf.alloc((size_t)n_pairs, s));
        VS_TRY(ksrc_buf.alloc((size_t)n_pairs, s));
        VS_TRY(filter_tiles.alloc((size_t)tiles, s));
        VS_CUDA_TRY(cudaMemsetAsync(filter_tiles.p, 0, (size_t)tiles * sizeof(unsigned long long), s));
        export_filter_kernel<<<(unsigned)tiles, kFilterThreads, 0, s>>>(
            d_left, d_right, n_pairs, n_left, n_right, d_left_code, d_right_code, kl_buf.p, kr_buf.p, ksrc_buf.p,
            filter_tiles.p, state.p);
        VS_LAUNCHED("export_filter", s);
        kl = kl_buf.p;
        kr = kr_buf.p;
        ksrc = ksrc_buf.p;
    }
    if (how == VS_HOW_INNER) {
        if (n_pairs > 0) {
            export_copy_kernel<<<grid_of(export_copy_kernel, n_pairs), 256, 0, s>>>(
                kl, kr, ksrc, state.p, capacity, d_out_left, d_out_right, d_out_src);
            VS_LAUNCHED("export_copy", s);
        }
        VS_TRY(read_state());
        return over_capacity((int64_t)h.kept);
    }
    // 2. the driving side: left rows, or right rows (pairs re-sorted by (right, left))
    const bool right = how == VS_HOW_RIGHT;
    const int64_t n_drive = right ? n_right : n_left;
    const int32_t* drive = right ? kr : kl;
    const int32_t* other = right ? kl : kr;
    const int64_t n_tiles = (n_drive + kTileRows - 1) / kTileRows;
    Scratch<uint64_t> keys;
    Scratch<uint32_t> perm, first, matched;
    VS_TRY(first.alloc((size_t)n_tiles + 1, s));
    VS_TRY(matched.alloc((size_t)n_tiles + 1, s));
    // 4. outer: right rows no pair reaches
    Scratch<uint32_t> missing, mpos;
    if (how == VS_HOW_OUTER && n_right > 0) {
        VS_TRY(missing.alloc((size_t)n_right, s));
        VS_TRY(mpos.alloc((size_t)n_right, s));
        VS_CUDA_TRY(cudaMemsetAsync(missing.p, 0, (size_t)n_right * sizeof(uint32_t), s));
        if (n_pairs > 0) {
            export_mark_kernel<<<grid_of(export_mark_kernel, n_pairs), 256, 0, s>>>(kr, n_right, missing.p, state.p);
            VS_LAUNCHED("export_mark", s);
        }
        export_flip_kernel<<<grid_of(export_flip_kernel, n_right), 256, 0, s>>>(missing.p, n_right);
        VS_LAUNCHED("export_flip", s);
        VS_TRY(exclusive_scan_u32(missing.p, mpos.p, n_right, &state.p->appended, s));
    }
    // 3. tiles of driving rows.  Pairs that are not sorted by (left, right), as they should be, are found by the
    // first attempt, which then writes nothing, and sorted for a second one.
    bool sorted = !right;
    for (int attempt = 0; attempt < 2; ++attempt) {
        ExportPairs pairs{drive, other, nullptr, nullptr, ksrc};
        if (!sorted) {
            VS_TRY(read_state());
            const int64_t m = h.kept;
            VS_TRY(keys.alloc((size_t)m, s));
            VS_TRY(perm.alloc((size_t)m, s));
            if (m > 0) {
                export_keys_kernel<<<grid_of(export_keys_kernel, m), 256, 0, s>>>(drive, other, m, keys.p, perm.p);
                VS_LAUNCHED("export_keys", s);
                VS_TRY(radix_sort_u64_u32(keys.p, perm.p, m, 64, s));
            }
            pairs = ExportPairs{nullptr, nullptr, keys.p, perm.p, ksrc};
            VS_CUDA_TRY(cudaMemsetAsync(&state.p->unsorted, 0, sizeof(uint32_t), s));
        }
        VS_CUDA_TRY(cudaMemsetAsync(first.p, 0, ((size_t)n_tiles + 1) * sizeof(uint32_t), s));
        VS_CUDA_TRY(cudaMemsetAsync(matched.p, 0, ((size_t)n_tiles + 1) * sizeof(uint32_t), s));
        if (n_pairs > 0 && n_tiles > 0) {
            export_bounds_kernel<<<grid_of(export_bounds_kernel, n_pairs), 256, 0, s>>>(pairs, n_drive, n_tiles,
                                                                                       first.p, matched.p, state.p);
            VS_LAUNCHED("export_bounds", s);
        }
        VS_TRY(exclusive_scan_u32(matched.p, matched.p, n_tiles, &state.p->distinct, s));
        if (n_tiles > 0) {
            const int64_t blocks = std::min<int64_t>(std::max<int64_t>(n_pairs / (n_tiles * kBlockPairs), 1), kTileBlocks);
            export_write_kernel<<<dim3((unsigned)n_tiles, (unsigned)blocks), kTileThreads, 0, s>>>(
                pairs, n_drive, first.p, matched.p, state.p, capacity, right ? d_out_right : d_out_left,
                right ? d_out_left : d_out_right, d_out_src);
            VS_LAUNCHED("export_write", s);
        }
        if (how == VS_HOW_OUTER && n_right > 0) {
            export_append_kernel<<<grid_of(export_append_kernel, n_right), 256, 0, s>>>(
                missing.p, mpos.p, n_right, state.p, n_drive, capacity, d_out_left, d_out_right, d_out_src);
            VS_LAUNCHED("export_append", s);
        }
        VS_TRY(read_state());
        if (!h.unsorted) break;
        sorted = false;
    }
    return over_capacity((int64_t)h.kept + (n_drive - (int64_t)h.distinct) + (int64_t)h.appended);
}

}  // extern "C"
