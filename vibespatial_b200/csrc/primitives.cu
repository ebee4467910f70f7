// Exclusive scan (reduce -> scan of block sums -> downsweep) and a stable
// LSD radix sort of (u32/u64 key, u32 value) items or (left, right) pairs,
// 8 or 9 bits per pass.
//
// Radix sort: one read of the keys counts every digit (rs_plan_kernel); then
// each pass reads and writes the items once (rs_pass_kernel): a tile gets the
// output position of its digit runs from the tiles before it while it runs (a
// decoupled look-back over per-tile counts) instead of from a histogram pass
// and a scan of their own.  Sorts of a few thousand items run in one block
// (rs_small_kernel).
#include <cuda_runtime.h>
#include <stdint.h>

#include "primitives.cuh"

namespace vs {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

template <class T>
__device__ __forceinline__ T warp_inclusive_scan(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread.
template <class T>
__device__ __forceinline__ void block_exclusive_scan(T v, T& excl) {
    __shared__ T warp_tot[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = warp_inclusive_scan(v);
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T w = lane < kScanThreads / 32 ? warp_tot[lane] : T(0);
        T wi = warp_inclusive_scan(w);
        if (lane < kScanThreads / 32) warp_tot[lane] = wi - w;
    }
    __syncthreads();
    excl = warp_tot[warp] + inc - v;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const T* __restrict__ in, int64_t n,
                                                                   T* __restrict__ sums) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    T acc = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
        if (i < n) acc += in[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __shared__ T ws[kScanThreads / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        T t = 0;
        for (int w = 0; w < kScanThreads / 32; ++w) t += ws[w];
        sums[blockIdx.x] = t;
    }
}

// Each thread owns kScanItems consecutive items.
template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_downsweep_kernel(const T* in, T* out, int64_t n,
                                                                      const T* __restrict__ offsets,
                                                                      T* __restrict__ d_total) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    T local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + k;
        v[k] = i < n ? in[i] : T(0);
        local += v[k];
    }
    T excl;
    block_exclusive_scan<T>(local, excl);
    T run = excl + (offsets ? offsets[blockIdx.x] : T(0));
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + k;
        if (i < n) out[i] = run;
        run += v[k];
        if (d_total && i == n - 1) *d_total = run;
    }
}

template <class T>
int exclusive_scan_impl(const T* in, T* out, int64_t n, T* d_total, cudaStream_t s) {
    if (n <= 0) {
        if (d_total) VS_CUDA_TRY(cudaMemsetAsync(d_total, 0, sizeof(T), s));
        return VS_OK;
    }
    const int64_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb > 0x7fffffff) {
        set_error("scan too large (%lld items)", (long long)n);
        return VS_E_ARG;
    }
    if (nb == 1) {
        scan_downsweep_kernel<T><<<1, kScanThreads, 0, s>>>(in, out, n, nullptr, d_total);
        VS_LAUNCHED("scan_downsweep", s);
        return VS_OK;
    }
    Scratch<T> sums;
    VS_TRY(sums.alloc((size_t)nb, s));
    scan_reduce_kernel<T><<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, sums.p);
    VS_LAUNCHED("scan_reduce", s);
    VS_TRY(exclusive_scan_impl<T>(sums.p, sums.p, nb, (T*)nullptr, s));
    scan_downsweep_kernel<T><<<(unsigned)nb, kScanThreads, 0, s>>>(in, out, n, sums.p, d_total);
    VS_LAUNCHED("scan_downsweep", s);
    return VS_OK;
}

// ------------------------------------------------------------------------
// Radix sort
// ------------------------------------------------------------------------
constexpr int kMaxDigits = 8;
constexpr int kRsThreads = 256;   // histogram blocks
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kPassThreads = 512;  // pass blocks: a thread a digit value at least
constexpr int kPassWarps = kPassThreads / 32;

// Which digits the passes sort by: digits that are the same in every key are
// left out.  Slot k of the pass launches sorts by digit[k] when k < n_slots.
// full: a pair sort by left and right (its order needs no fixing).
struct SortPlan {
    uint32_t n_slots;
    uint32_t full;
    uint32_t max_left;
    uint32_t digit[kMaxDigits];
};

// How a pair sort orders equal left rows: by digits of right too, or by a last
// pass over the (short) runs of equal left rows, or the plan decides.
enum : int { kPairsFull = 0, kPairsRuns = 1, kPairsAuto = 2 };
// Pairs a left row may have on average for the run pass to be used: with up to
// 8 it reads a handful of neighbours, and saves the passes over right's digits
// (half of them for 20-bit rows).
constexpr int64_t kRunMean = 8;
constexpr int kRunMax = 1024;  // pairs of a run behind the tile it begins in that the run pass still orders

// One sort.  The items are (key, value) arrays, or (left, right) pairs whose
// key is left << rbits | right and which carry no value.  Arrays: slot 0 reads
// the caller's, the last slot writes them; pairs: slot 0 reads the caller's,
// the run pass writes them.  The slots between alternate between two buffers.
template <class K>
struct SortArgs {
    K* keys;            // null: pairs
    uint32_t* vals;
    int32_t* left;
    int32_t* right;
    int rbits;
    int pairs_mode;
    K* kbuf[2];
    uint32_t* vbuf[2];
    int64_t n;
    int shift[kMaxDigits];
    int n_digits;
    int n_right;        // pairs: digits [0, n_right) are right's
    uint32_t* hist;     // [n_digits][radix] counts, then exclusive sums
    uint32_t* ticket;   // [0] histogram blocks done, [1 + slot] tiles handed out
    SortPlan* plan;
    unsigned long long* too_long;  // pairs by runs: gets bit 2 (nullable)
    int64_t n_tiles;
};

template <class K>
__device__ __forceinline__ K sort_key(const K* keys, const int32_t* left, const int32_t* right, int rbits, int64_t i) {
    if (keys) return keys[i];
    return (K)(((uint64_t)(uint32_t)left[i] << rbits) | (uint64_t)(uint32_t)right[i]);
}
template <class K>
__device__ __forceinline__ K sort_key(const SortArgs<K>& a, const K* keys, int64_t i) {
    return sort_key(keys, a.left, a.right, a.rbits, i);
}

// Every digit's histogram in one read of the keys; the last block to finish
// turns them into exclusive sums and writes the plan.  The counters are
// shared-memory increments.
template <class K, int kBits>
__global__ void __launch_bounds__(kRsThreads) rs_plan_kernel(const SortArgs<K> a) {
    constexpr int kRadix = 1 << kBits, kPer = kRadix / kRsThreads;
    __shared__ uint32_t h[kMaxDigits][kRadix];
    __shared__ uint32_t s_one[kMaxDigits];
    __shared__ uint32_t s_sum[kRsWarps];
    __shared__ uint32_t s_max;
    __shared__ bool s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < a.n_digits * kRadix; i += kRsThreads) (&h[0][0])[i] = 0;
    if (tid == 0) s_max = 0;
    __syncthreads();
    uint32_t max_left = 0;
    for (int64_t i = (int64_t)blockIdx.x * kRsThreads + tid; i < a.n; i += (int64_t)gridDim.x * kRsThreads) {
        const K k = sort_key(a, a.keys, i);
        if (a.pairs_mode == kPairsAuto) max_left = max(max_left, (uint32_t)((uint64_t)k >> a.rbits));
#pragma unroll
        for (int d = 0; d < kMaxDigits; ++d)
            if (d < a.n_digits) atomicAdd(&h[d][(unsigned)(k >> a.shift[d]) & (kRadix - 1)], 1u);
    }
    if (a.pairs_mode == kPairsAuto) atomicMax(&s_max, max_left);
    __syncthreads();
    for (int i = tid; i < a.n_digits * kRadix; i += kRsThreads)
        if (uint32_t c = (&h[0][0])[i]) atomicAdd(&a.hist[i], c);
    if (tid == 0 && s_max) atomicMax(&a.plan->max_left, s_max);
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&a.ticket[0], 1u) == gridDim.x - 1;
    if (tid < kMaxDigits) s_one[tid] = 0;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int d = 0; d < a.n_digits; ++d) {
        uint32_t c[kPer], t = 0;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            c[u] = __ldcg(&a.hist[d * kRadix + tid * kPer + u]);
            if ((int64_t)c[u] == a.n) s_one[d] = 1;  // every key has this digit
            t += c[u];
        }
        const uint32_t inc = warp_inclusive_scan(t);
        if (lane == 31) s_sum[warp] = inc;
        __syncthreads();
        uint32_t before = inc - t;
        for (int w = 0; w < warp; ++w) before += s_sum[w];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            a.hist[d * kRadix + tid * kPer + u] = before;
            before += c[u];
        }
        __syncthreads();
    }
    if (tid == 0) {
        const bool pairs = a.keys == nullptr;
        const bool full = a.pairs_mode == kPairsFull ||
                          (a.pairs_mode == kPairsAuto && a.n > kRunMean * ((int64_t)__ldcg(&a.plan->max_left) + 1));
        uint32_t k = 0;
        for (int d = full ? 0 : a.n_right; d < a.n_digits; ++d)
            if (!s_one[d]) a.plan->digit[k++] = (uint32_t)d;
        // pairs go through a buffer at least once; one slot on arrays would read and write them at once
        if (pairs && k == 0) a.plan->digit[k++] = (uint32_t)(a.n_digits - 1);
        if (!pairs && k == 1) a.plan->digit[k++] = a.plan->digit[0];
        a.plan->full = full ? 1u : 0u;
        a.plan->n_slots = k;
    }
}

// Lanes whose digit equals this lane's: a ballot a bit.  (__match_any_sync
// steps through the distinct digits one after another: a pass over 10M pairs
// took half as long again with it.)
template <int kBits>
__device__ __forceinline__ unsigned same_digit(unsigned d) {
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < kBits; ++b) {
        const bool on = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        peers &= on ? m : ~m;
    }
    return peers;
}

// Stable ranks of R rounds of 32 keys of a warp among the warp's keys of the
// same digit: rank[r] counts the warp's earlier ones; cnt (the warp's own
// counters, zeroed) ends as the warp's digit counts.
template <class K, int kBits, int R>
__device__ __forceinline__ void warp_rank(const K (&k)[R], int shift, uint32_t* cnt, uint32_t (&rank)[R]) {
    const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const unsigned d = (unsigned)(k[r] >> shift) & ((1u << kBits) - 1u);
        const unsigned peers = same_digit<kBits>(d);
        const uint32_t before = cnt[d];
        __syncwarp();
        rank[r] = before + __popc(peers & lt);
        if ((peers & lt) == 0u) cnt[d] = before + __popc(peers);
        __syncwarp();
    }
}

// A tile state is one word, so relaxed accesses carry it whole.
__device__ __forceinline__ uint32_t load_state(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long load_state(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_state(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void store_state(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Polls of earlier tiles before a tile counts their keys itself (a build may lower it to test that).
#ifndef VS_SORT_WAIT_LIMIT
#define VS_SORT_WAIT_LIMIT (1 << 20)
#endif
constexpr int kWaitLimit = VS_SORT_WAIT_LIMIT;
// Earlier tiles whose states a tile reads at once: the tiles of a pass's first
// wave start together and have only counts, no sums, to read from one another.
constexpr int kLookBack = 8;

template <class K, bool kVals, int kBits, int R>
struct PassShared {
    static constexpr int kRadix = 1 << kBits;
    static constexpr int T = kPassThreads * R;
    uint32_t wcnt[kPassWarps][kRadix];
    uint32_t start[kRadix];  // tile-local start of a digit
    unsigned long long off[kRadix];  // output position of a digit's run minus its tile-local start
    uint32_t sum[kPassWarps];
    uint32_t tile;
    alignas(16) K key[T];
    uint32_t val[kVals ? T : 1];
};

// Keys of a digit value among the first n of a pass's input, by one thread.  A
// tile that has waited kWaitLimit polls for an earlier one counts that tile's
// keys, and those before it, this way: the input is complete before the pass
// starts, so the positions are right whatever became of the wait.
template <class K>
__device__ __noinline__ uint32_t count_digit(const K* keys, const int32_t* left, const int32_t* right, int rbits,
                                             int64_t n, int shift, unsigned mask, unsigned digit) {
    uint32_t c = 0;
    for (int64_t i = 0; i < n; ++i)
        c += ((unsigned)(sort_key(keys, left, right, rbits, i) >> shift) & mask) == digit ? 1u : 0u;
    return c;
}

// One slot of the sort: the tiles are taken in order (a ticket), so every tile
// before a running one is running or done.  A tile ranks its keys (warp by
// warp, no block barrier in between), publishes its digit counts, stages the
// keys in digit order in shared memory, sums the counts of the tiles before
// it (each publishes its counts, then its inclusive sums, as value << 2 |
// state in one word: S), and writes the digit runs.  Keys are read and
// written once a pass.  A wait that runs out ends in a count (count_digit).
//
// Bound by instruction issue (the ranks: a ballot a bit) at two blocks an SM.
// 12.2M pairs with 26 and 20 bits of rows: 94 us the first pass, which need
// not be stable, 117 us each of the two others (9-bit digits), 440 us the whole
// sort with the plan and the run pass; a histogram, a scan and a scatter for
// each of six 8-bit digits took 1160 us.
template <class K, bool kVals, class S, int kBits, int R, bool kStable>
__global__ void __launch_bounds__(kPassThreads) rs_pass_kernel(const SortArgs<K> a, int slot, S* __restrict__ status) {
    using Shared = PassShared<K, kVals, kBits, R>;
    constexpr int T = Shared::T, kRadix = Shared::kRadix;
    extern __shared__ __align__(16) unsigned char s_raw[];
    Shared& sm = *reinterpret_cast<Shared*>(s_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_slots = (int)a.plan->n_slots;
    if (slot >= n_slots) return;
    const int digit = (int)a.plan->digit[slot];
    const int shift = a.shift[digit];
    const K* kin = slot == 0 ? a.keys : a.kbuf[(slot - 1) & 1];
    const uint32_t* vin = slot == 0 ? a.vals : a.vbuf[(slot - 1) & 1];
    if (tid == 0) sm.tile = atomicAdd(&a.ticket[1 + slot], 1u);
    constexpr int kCounters = kStable ? kPassWarps : 1;  // sets of digit counters: a warp's own, or the block's
    for (int i = tid; i < kCounters * kRadix / 4; i += kPassThreads)
        reinterpret_cast<uint4*>(&sm.wcnt[0][0])[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const int64_t tile = sm.tile;
    const int64_t tile0 = tile * T;
    const int count = (int)(a.n - tile0 < T ? a.n - tile0 : T);
    const int at = warp * 32 * R + lane;
    K k[R];
    uint32_t v[R], rank[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = at + r * 32;
        k[r] = ~(K)0;  // past the end: the last digit, ranked behind the tile's own keys
        v[r] = 0;
        if (j < count) {
            k[r] = sort_key(a, kin, tile0 + j);
            if (kVals) v[r] = vin[tile0 + j];
        }
    }
    if constexpr (kStable) {
        warp_rank<K, kBits, R>(k, shift, sm.wcnt[warp], rank);
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) rank[r] = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)  // (a key past the end is not counted and not placed)
            if (at + r * 32 < count) rank[r] = atomicAdd(&sm.wcnt[0][(unsigned)(k[r] >> shift) & (unsigned)(kRadix - 1)], 1u);
    }
    __syncthreads();
    // thread t < radix owns digit t: per-warp starts, the tile's count, its scan
    uint32_t total = 0, own = 0, before = 0;
    S* st = status + tile * kRadix + tid;
    if (tid < kRadix) {
#pragma unroll
        for (int w = 0; w < kCounters; ++w) {
            const uint32_t c = sm.wcnt[w][tid];
            sm.wcnt[w][tid] = total;
            total += c;
        }
        own = total - (kStable && tid == kRadix - 1 ? (uint32_t)(T - count) : 0u);
        if (tile > 0) store_state(st, ((S)own << 2) | (S)1);
        const uint32_t inc = warp_inclusive_scan(total);
        if (lane == 31) sm.sum[warp] = inc;
        before = inc - total;
    }
    __syncthreads();
    if (tid < kRadix) {
        for (int w = 0; w < warp; ++w) before += sm.sum[w];
        sm.start[tid] = before;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const unsigned d = (unsigned)(k[r] >> shift) & (unsigned)(kRadix - 1);
        if (!kStable && at + r * 32 >= count) break;
        const uint32_t pos = sm.start[d] + (kStable ? sm.wcnt[warp][d] : 0u) + rank[r];
        sm.key[pos] = k[r];
        if (kVals) sm.val[pos] = v[r];
    }
    if (tid < kRadix) {
        S sum = 0;
        int polls = 0;
        for (int64_t t = tile - 1; t >= 0;) {
            // kLookBack states at once: the loads' latencies overlap
            S w[kLookBack];
#pragma unroll
            for (int j = 0; j < kLookBack; ++j) w[j] = t >= j ? load_state(status + (t - j) * kRadix + tid) : (S)2;
            bool ready = true, done = false;
#pragma unroll
            for (int j = 0; j < kLookBack; ++j) {
                ready = ready && (w[j] & 3) != 0;
                if (ready && !done) {
                    sum += w[j] >> 2;
                    done = (w[j] & 3) == 2;
                    --t;
                }
            }
            if (done) break;
            if (!ready) {
                // wait for the one state that is missing, without flooding L2
                while ((load_state(status + t * kRadix + tid) & 3) == 0 && ++polls < kWaitLimit) __nanosleep(40);
                if (polls >= kWaitLimit) {
                    sum += count_digit(kin, a.left, a.right, a.rbits, (t + 1) * T, shift, kRadix - 1u, (unsigned)tid);
                    break;
                }
            }
        }
        store_state(st, ((sum + (S)own) << 2) | (S)2);
        sm.off[tid] = (unsigned long long)a.hist[digit * kRadix + tid] + sum - before;
    }
    __syncthreads();
    const bool arrays_last = a.keys && slot == n_slots - 1;
    K* kout = arrays_last ? a.keys : a.kbuf[slot & 1];
    uint32_t* vout = arrays_last ? a.vals : a.vbuf[slot & 1];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = tid + r * kPassThreads;
        if (j >= count) break;
        const K key = sm.key[j];
        const unsigned long long pos = sm.off[(unsigned)(key >> shift) & (unsigned)(kRadix - 1)] + (unsigned)j;
        kout[pos] = key;
        if (kVals) vout[pos] = sm.val[j];
    }
}

// The pairs, sorted by left, back to the caller's arrays, each run of equal
// left rows in the order of its right rows.  A run belongs to the block whose
// tile it begins in, which holds it to its end, up to kRunMax pairs beyond the
// tile; a run that goes on longer is left as it is and reported (bit 2 of
// *too_long): such pairs are sorted by right's digits instead.
//
// Short runs: each pair counts the smaller ones of its run (equal ones in their
// order).  A tile with a run longer than kRunLong, or with many longer than
// kRunShort, sorts its pairs by run and right row in shared memory: the count
// is quadratic in the run, the sort is not.  Whole sorts of 12M pairs (14M for
// runs of 1000), us, with every tile counting / as it is: runs of 32 pairs
// 664 / 658, 40 736 / 565, 64 933 / 629, 100 1121 / 568, 400 2711 / 572, 1000
// 6914 / 686; with runs of 2000, and so a second sort, 10554 / 1241.  (Passes
// over all digits, each with a histogram and a scan of its own, took 990 to
// 1130.)
constexpr int kRunThreads = 256, kRunItems = 8, kRunTile = kRunThreads * kRunItems, kRunWarps = kRunThreads / 32;
constexpr int kRunHeld = kRunTile + kRunMax;
constexpr int kRunRounds = kRunHeld / kRunThreads;
constexpr int kRunShort = 24;
constexpr int kRunLong = 192;
static_assert(kRunHeld % kRunThreads == 0 && kRunHeld <= 0xffff, "a run's number fits 16 bits");
static_assert(kRunLong + 16 <= kRunThreads, "the count looks at a tile and as many pairs behind it as it has threads");

struct RunShared {
    uint32_t left[kRunHeld], right[kRunHeld];
    uint16_t run[kRunHeld];
    uint32_t cnt[kRunWarps][256];
    uint32_t sum[kRunWarps];
    int first, last, behind;
    bool goes_on, long_before;  // the tile's first run begins before it; before the tile before it
};

// Sort the m pairs held from h0 on by (run, right): right rows only, a place's
// left row stays what it is.  Whole block.
__device__ __noinline__ void sort_held_runs(RunShared& sm, int h0, int m, int rbits) {
    constexpr unsigned kAll = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int at = warp * 32 * kRunRounds + lane;
    uint32_t right[kRunRounds], run[kRunRounds], rank[kRunRounds];
    // the number of a pair's run among those held
    uint32_t heads = 0;
#pragma unroll
    for (int r = 0; r < kRunRounds; ++r) {
        const int q = at + 32 * r;
        const unsigned b = __ballot_sync(kAll, q > 0 && q < m && sm.left[h0 + q] != sm.left[h0 + q - 1]);
        run[r] = heads + __popc(b & (kAll >> (31 - lane)));
        heads += __popc(b);  // warp-uniform
        right[r] = q < m ? sm.right[h0 + q] : kAll;  // (past the end: behind every pair)
    }
    if (lane == 0) sm.sum[warp] = heads;
    __syncthreads();
    uint32_t base = 0, runs = 0;
    for (int w = 0; w < kRunWarps; ++w) {
        base += w < warp ? sm.sum[w] : 0u;
        runs += sm.sum[w];
    }
#pragma unroll
    for (int r = 0; r < kRunRounds; ++r) run[r] = at + 32 * r < m ? base + run[r] : 0xffffu;
    const int run_passes = runs == 0 ? 0 : runs < 0xffu ? 1 : 2;
    for (int pass = -((rbits + 7) / 8); pass < run_passes; ++pass) {
        const bool by_run = pass >= 0;
        const int shift = by_run ? 8 * pass : 8 * (pass + (rbits + 7) / 8);
        __syncthreads();
        for (int i = tid; i < kRunWarps * 256; i += kRunThreads) (&sm.cnt[0][0])[i] = 0;
        __syncthreads();
        if (by_run) warp_rank<uint32_t, 8, kRunRounds>(run, shift, sm.cnt[warp], rank);
        else warp_rank<uint32_t, 8, kRunRounds>(right, shift, sm.cnt[warp], rank);
        __syncthreads();
        uint32_t total = 0;  // of digit tid
        for (int w = 0; w < kRunWarps; ++w) {
            const uint32_t c = sm.cnt[w][tid];
            sm.cnt[w][tid] = total;
            total += c;
        }
        const uint32_t inc = warp_inclusive_scan(total);
        if (lane == 31) sm.sum[warp] = inc;
        __syncthreads();
        uint32_t start = inc - total;
        for (int w = 0; w < warp; ++w) start += sm.sum[w];
        for (int w = 0; w < kRunWarps; ++w) sm.cnt[w][tid] += start;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRunRounds; ++r) {
            const unsigned d = ((by_run ? run[r] : right[r]) >> shift) & 255u;
            const uint32_t pos = sm.cnt[warp][d] + rank[r];
            if (pos < (uint32_t)m) {  // (those past the end come last)
                sm.right[h0 + pos] = right[r];
                sm.run[pos] = (uint16_t)run[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRunRounds; ++r) {
            const int q = at + 32 * r;
            right[r] = q < m ? sm.right[h0 + q] : kAll;
            run[r] = q < m ? (uint32_t)sm.run[q] : 0xffffu;
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kRunThreads, 5) rs_runs_kernel(const SortArgs<uint64_t> a) {
    __shared__ RunShared sm;
    const uint64_t* __restrict__ key = a.kbuf[(a.plan->n_slots - 1) & 1];
    const uint64_t rmask = (1ull << a.rbits) - 1ull;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t tile0 = (int64_t)blockIdx.x * kRunTile;
    const int count = (int)(a.n - tile0 < kRunTile ? a.n - tile0 : kRunTile);
    if (a.plan->full != 0) {  // sorted by right too
        for (int j = tid; j < count; j += kRunThreads) {
            const uint64_t k = key[tile0 + j];
            a.left[tile0 + j] = (int32_t)(k >> a.rbits);
            a.right[tile0 + j] = (int32_t)(k & rmask);
        }
        return;
    }
    for (int j = tid; j < count; j += kRunThreads) {
        const uint64_t k = key[tile0 + j];
        sm.left[j] = (uint32_t)(k >> a.rbits);
        sm.right[j] = (uint32_t)(k & rmask);
    }
    if (tid == 0) {
        const uint32_t l0 = (uint32_t)(key[tile0] >> a.rbits);
        sm.goes_on = tile0 > 0 && (uint32_t)(key[tile0 - 1] >> a.rbits) == l0;
        sm.long_before = tile0 > kRunTile && (uint32_t)(key[tile0 - kRunTile - 1] >> a.rbits) == l0;
        sm.first = count;
        sm.last = -1;
    }
    if (warp == 1) {  // pairs of the tile's last run behind it (more than kRunMax: any such number)
        const int64_t end = tile0 + count;
        const uint32_t l1 = (uint32_t)(key[end - 1] >> a.rbits);
        int behind = 0;
        for (unsigned m = 0xffffffffu; m == 0xffffffffu && behind <= kRunMax;) {
            const int64_t i = end + behind + lane;
            m = __ballot_sync(0xffffffffu, i < a.n && (uint32_t)(key[i] >> a.rbits) == l1);
            behind += m == 0xffffffffu ? 32 : __ffs(~m) - 1;
        }
        if (lane == 0) sm.behind = behind;
    }
    __syncthreads();
    // the first and the last run that begin in the tile
    int first = count, last = -1;
#pragma unroll
    for (int u = 0; u < kRunItems; ++u) {
        const int j = tid + u * kRunThreads;
        if (j < count && (j > 0 ? sm.left[j] != sm.left[j - 1] : !sm.goes_on)) {
            first = min(first, j);
            last = j;
        }
    }
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) {
        if (first < count) atomicMin(&sm.first, first);
        if (last >= 0) atomicMax(&sm.last, last);
    }
    __syncthreads();
    const int h0 = sm.first, hl = sm.last, behind = sm.behind;
    const bool first_long = sm.goes_on && (h0 > kRunMax || sm.long_before);
    const bool last_long = hl >= 0 && behind > kRunMax;
    const int end = hl < 0 ? h0 : last_long ? hl : count + behind;  // the tile's own runs: [h0, end)
    if (!last_long && hl >= 0)
        for (int j = count + tid; j < end; j += kRunThreads) {
            const uint64_t k = key[tile0 + j];
            sm.left[j] = (uint32_t)(k >> a.rbits);
            sm.right[j] = (uint32_t)(k & rmask);
        }
    if (first_long || last_long) {
        for (int j = tid; j < count; j += kRunThreads)
            if (j < h0 ? first_long : j >= end) {
                a.left[tile0 + j] = (int32_t)sm.left[j];
                a.right[tile0 + j] = (int32_t)sm.right[j];
            }
        if (tid == 0 && a.too_long) atomicOr(a.too_long, 4ull);
    }
    __syncthreads();
    // by samples: a run longer than kRunLong, or a quarter of the pairs with more than kRunShort of their run behind them
    const int j = h0 + 16 * tid;
    const bool longer = j + kRunShort < end && sm.left[j] == sm.left[j + kRunShort];
    const int samples = (end - h0 + 15) / 16;
    const bool one = longer && j + kRunLong < end && sm.left[j] == sm.left[j + kRunLong];
    const int many = __syncthreads_count(longer);
    if (__syncthreads_or(one) || 4 * many > samples) {
        sort_held_runs(sm, h0, end - h0, a.rbits);
        for (int i = h0 + tid; i < end; i += kRunThreads) {
            a.left[tile0 + i] = (int32_t)sm.left[i];
            a.right[tile0 + i] = (int32_t)sm.right[i];
        }
        return;
    }
#pragma unroll
    for (int u = 0; u < kRunItems + 1; ++u) {
        const int j0 = tid + u * kRunThreads;  // (the last run has kRunLong + 16 pairs at most)
        if (j0 < h0 || j0 >= end) continue;
        const uint32_t l = sm.left[j0], r = sm.right[j0];
        int move = 0;  // larger ones before move behind, smaller ones behind move before
        for (int i = j0 - 1; i >= h0 && sm.left[i] == l; --i) move -= sm.right[i] > r ? 1 : 0;
        for (int i = j0 + 1; i < end && sm.left[i] == l; ++i) move += sm.right[i] < r ? 1 : 0;
        a.left[tile0 + j0 + move] = (int32_t)l;
        a.right[tile0 + j0 + move] = (int32_t)r;
    }
}

// A sort of at most kSmallSort items in one block: every pass in shared
// memory, one launch instead of two plus one a digit.
constexpr int kRadix = 256;
constexpr int kSmallThreads = 1024;
constexpr int kSmallRounds = 8;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int64_t kSmallSort = (int64_t)kSmallThreads * kSmallRounds;

template <class K, bool kVals, int R>
__global__ void __launch_bounds__(kSmallThreads) rs_small_kernel(const SortArgs<K> a) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    K* s_key = reinterpret_cast<K*>(s_raw);
    uint32_t* s_val = reinterpret_cast<uint32_t*>(s_key + kSmallThreads * R);
    uint32_t* wcnt = s_val + (kVals ? kSmallThreads * R : 0);
    __shared__ uint32_t s_part[4][kRadix];
    __shared__ uint32_t s_start[kRadix];
    __shared__ uint32_t s_sum[kRadix / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = (int)a.n;
    const int at = warp * 32 * R + lane;
    K k[R];
    uint32_t v[R], rank[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = at + r * 32;
        k[r] = ~(K)0;  // past the end: ranked behind every item
        v[r] = 0;
        if (j < n) {
            k[r] = sort_key(a, a.keys, j);
            if (kVals) v[r] = a.vals[j];
        }
    }
    for (int digit = 0; digit < a.n_digits; ++digit) {
        const int shift = a.shift[digit];
        for (int i = tid; i < kSmallWarps * kRadix; i += kSmallThreads) wcnt[i] = 0;
        __syncthreads();
        warp_rank<K, 8, R>(k, shift, wcnt + warp * kRadix, rank);
        __syncthreads();
        // digit tid % 256, warps [8 q, 8 q + 8): counts to starts within the quarter
        const int q = tid >> 8, d0 = tid & (kRadix - 1);
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            uint32_t* c = &wcnt[(q * 8 + w) * kRadix + d0];
            const uint32_t x = *c;
            *c = total;
            total += x;
        }
        s_part[q][d0] = total;
        __syncthreads();
        if (tid < kRadix) {
            uint32_t t = 0;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const uint32_t x = s_part[w][tid];
                s_part[w][tid] = t;
                t += x;
            }
            const uint32_t inc = warp_inclusive_scan(t);
            if (lane == 31) s_sum[warp] = inc;
            s_start[tid] = inc - t;
        }
        __syncthreads();
        if (tid < kRadix) {
            uint32_t before = 0;
            for (int w = 0; w < warp; ++w) before += s_sum[w];
            s_start[tid] += before;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned d = (unsigned)(k[r] >> shift) & 0xffu;
            const uint32_t pos = s_start[d] + s_part[warp >> 3][d] + wcnt[warp * kRadix + d] + rank[r];
            s_key[pos] = k[r];
            if (kVals) s_val[pos] = v[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            k[r] = s_key[at + r * 32];
            if (kVals) v[r] = s_val[at + r * 32];
        }
    }
    const uint32_t rmask = (uint32_t)((1ull << a.rbits) - 1ull);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = at + r * 32;
        if (j >= n) continue;
        if (a.keys) {
            a.keys[j] = k[r];
            if (kVals) a.vals[j] = v[r];
        } else {
            a.left[j] = (int32_t)((uint64_t)k[r] >> a.rbits);
            a.right[j] = (int32_t)((uint32_t)k[r] & rmask);
        }
    }
}

template <class K, bool kVals, int R>
int launch_small_sort(const SortArgs<K>& a, cudaStream_t s) {
    constexpr size_t smem = (size_t)kSmallThreads * R * (sizeof(K) + (kVals ? sizeof(uint32_t) : 0)) +
                            (size_t)kSmallWarps * kRadix * sizeof(uint32_t);
    auto* kernel = rs_small_kernel<K, kVals, R>;
    VS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<1, kSmallThreads, smem, s>>>(a);
    VS_LAUNCHED("rs_small", s);
    return VS_OK;
}

template <class K, bool kVals, class S, int kBits, int R>
int run_passes(SortArgs<K>& a, cudaStream_t s) {
    constexpr int kRadix = 1 << kBits;
    constexpr int64_t T = (int64_t)kPassThreads * R;
    a.n_tiles = (a.n + T - 1) / T;
    const bool pairs = a.keys == nullptr;
    int slots = pairs && a.pairs_mode == kPairsRuns ? a.n_digits - a.n_right : a.n_digits;
    if (!pairs && slots < 2) slots = 2;
    // one zeroed block: tickets, plan, histograms, the slots' tile states
    constexpr size_t kHead = 64 * sizeof(uint32_t);
    const size_t hist_b = (size_t)a.n_digits * kRadix * sizeof(uint32_t);
    const size_t status_b = (size_t)a.n_tiles * kRadix * sizeof(S);
    Scratch<char> state;
    Scratch<K> k0, k1;
    Scratch<uint32_t> v0, v1;
    const bool two = slots > (pairs ? 1 : 2);
    VS_TRY(state.alloc(kHead + hist_b + (size_t)slots * status_b, s));
    VS_TRY(k0.alloc((size_t)a.n, s));
    if (two) VS_TRY(k1.alloc((size_t)a.n, s));
    if (kVals) {
        VS_TRY(v0.alloc((size_t)a.n, s));
        if (two) VS_TRY(v1.alloc((size_t)a.n, s));
    }
    a.kbuf[0] = k0.p;
    a.kbuf[1] = k1.p;
    a.vbuf[0] = v0.p;
    a.vbuf[1] = v1.p;
    a.ticket = reinterpret_cast<uint32_t*>(state.p);
    a.plan = reinterpret_cast<SortPlan*>(a.ticket + 16);
    a.hist = a.ticket + 64;
    S* status = reinterpret_cast<S*>(state.p + kHead + hist_b);
    VS_CUDA_TRY(cudaMemsetAsync(state.p, 0, kHead + hist_b + (size_t)slots * status_b, s));
    rs_plan_kernel<K, kBits><<<grid_for((a.n + 15) / 16, kRsThreads, 8), kRsThreads, 0, s>>>(a);
    VS_LAUNCHED("rs_plan", s);
    constexpr size_t smem = sizeof(PassShared<K, kVals, kBits, R>);
    for (int k = 0; k < slots; ++k) {
        // the order the pairs come in does not matter, so their first pass need not keep it
        auto* kernel = k == 0 && !kVals ? rs_pass_kernel<K, kVals, S, kBits, R, kVals>
                                        : rs_pass_kernel<K, kVals, S, kBits, R, true>;
        VS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<(unsigned)a.n_tiles, kPassThreads, smem, s>>>(a, k, status + (size_t)k * a.n_tiles * kRadix);
        VS_LAUNCHED("rs_pass", s);
    }
    if constexpr (!kVals) {
        rs_runs_kernel<<<(unsigned)((a.n + kRunTile - 1) / kRunTile), kRunThreads, 0, s>>>(a);
        VS_LAUNCHED("rs_runs", s);
    }
    return VS_OK;
}

// Keys a thread of a pass holds: 8 (6 with values behind 64-bit keys); 2 up to
// this many items, so that a small sort spreads over the SMs and its tiles
// take less time each.
constexpr int64_t kFewItems = (int64_t)kNumSMs * kPassThreads * 4;

template <class K, bool kVals, int kBits>
int run_sort(SortArgs<K>& a, cudaStream_t s) {
    constexpr int R = sizeof(K) + (kVals ? 4 : 0) > 8 ? 6 : 8;
    if (a.n <= kFewItems) return run_passes<K, kVals, uint32_t, kBits, 2>(a, s);
    // tile states hold sums below 2^30 in 32-bit words
    if (a.n < (1ll << 30)) return run_passes<K, kVals, uint32_t, kBits, R>(a, s);
    return run_passes<K, kVals, unsigned long long, kBits, R>(a, s);
}

int check_count(int64_t n) {
    if (n <= 0xffffffffLL) return VS_OK;
    set_error("radix sort supports at most 2^32-1 items (got %lld)", (long long)n);
    return VS_E_ARG;
}

// Digits of `bits` bits each over key bits [begin, end), the last one ending
// at or past `end`; one that would reach past the key's top bit overlaps the
// one before it instead, which still sorts stably.
template <class K>
void add_digits(SortArgs<K>& a, int begin, int end, int bits) {
    const int max_bits = (int)(8 * sizeof(K));
    for (int sh = begin; sh < end; sh += bits) a.shift[a.n_digits++] = sh + bits > max_bits ? max_bits - bits : sh;
}

template <class K>
int sort_arrays(SortArgs<K>& a, int begin_bit, int end_bit, cudaStream_t s) {
    if (a.n <= 1) return VS_OK;
    VS_TRY(check_count(a.n));
    const int max_bits = (int)(8 * sizeof(K));
    if (end_bit <= 0 || end_bit > max_bits) end_bit = max_bits;
    if (begin_bit < 0 || begin_bit >= end_bit) begin_bit = 0;
    add_digits(a, begin_bit, end_bit, 8);
    if (a.n <= 2 * kSmallThreads) return launch_small_sort<K, true, 2>(a, s);
    if (a.n <= kSmallSort) return launch_small_sort<K, true, kSmallRounds>(a, s);
    return run_sort<K, true, 8>(a, s);
}

}  // namespace

int exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* d_total, cudaStream_t s) {
    return exclusive_scan_impl<uint32_t>(in, out, n, d_total, s);
}
int exclusive_scan_u64(const uint64_t* in, uint64_t* out, int64_t n, uint64_t* d_total, cudaStream_t s) {
    return exclusive_scan_impl<uint64_t>(in, out, n, d_total, s);
}

int radix_sort_u64_u32(uint64_t* keys, uint32_t* vals, int64_t n, int key_bits, cudaStream_t s, int begin_bit) {
    SortArgs<uint64_t> a{};
    a.keys = keys;
    a.vals = vals;
    a.n = n;
    return sort_arrays(a, begin_bit, key_bits, s);
}

int radix_sort_u32_u32(uint32_t* keys, uint32_t* vals, int64_t n, int key_bits, cudaStream_t s, int begin_bit) {
    SortArgs<uint32_t> a{};
    a.keys = keys;
    a.vals = vals;
    a.n = n;
    return sort_arrays(a, begin_bit, key_bits, s);
}

int radix_sort_pairs(int32_t* left, int32_t* right, int64_t n, int left_bits, int right_bits, int64_t n_left,
                     bool by_runs, cudaStream_t s, unsigned long long* too_long) {
    if (n <= 1) return VS_OK;
    VS_TRY(check_count(n));
    SortArgs<uint64_t> a{};
    a.left = left;
    a.right = right;
    a.rbits = right_bits;
    a.n = n;
    a.too_long = too_long;
    if (n <= kSmallSort) {
        add_digits(a, 0, left_bits + right_bits, 8);
        return n <= 2 * kSmallThreads ? launch_small_sort<uint64_t, false, 2>(a, s)
                                      : launch_small_sort<uint64_t, false, kSmallRounds>(a, s);
    }
    a.pairs_mode = !by_runs ? kPairsFull : n_left <= 0 ? kPairsAuto : n > kRunMean * n_left ? kPairsFull : kPairsRuns;
    if (a.pairs_mode == kPairsRuns) {
        // 9-bit digits where they save a pass over left's bits
        if ((left_bits + 8) / 9 < (left_bits + 7) / 8) {
            add_digits(a, right_bits, right_bits + left_bits, 9);
            return run_sort<uint64_t, false, 9>(a, s);
        }
        add_digits(a, right_bits, right_bits + left_bits, 8);
        return run_sort<uint64_t, false, 8>(a, s);
    }
    if (a.pairs_mode == kPairsAuto) {
        // right's digits apart from left's: the plan may drop them
        add_digits(a, 0, right_bits, 8);
        a.n_right = a.n_digits;
        add_digits(a, right_bits, right_bits + left_bits, 8);
    } else {
        add_digits(a, 0, left_bits + right_bits, 8);
    }
    return run_sort<uint64_t, false, 8>(a, s);
}

}  // namespace vs
