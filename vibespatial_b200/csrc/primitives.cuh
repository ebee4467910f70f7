// In-house device primitives (scan, radix sort) and stream-ordered scratch.
//
// The reference calls CCCL for these (exclusive_sum, radix sort_pairs,
// select, lower/upper_bound: src/vibespatial/cuda/cccl_primitives.py:523-1167);
// the build forbids CCCL/CUB on the hot path, so they are written here.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "vs_common.cuh"

namespace vs {

// Stream-ordered scratch buffer (cudaMallocAsync / cudaFreeAsync on the
// context stream; the device pool keeps freed blocks, so steady-state calls do
// not reach the driver).
template <class T>
struct Scratch {
    T* p = nullptr;
    cudaStream_t s = nullptr;
    Scratch() = default;
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    int alloc(size_t n, cudaStream_t stream) {
        release();
        s = stream;
        if (n == 0) n = 1;
        cudaError_t e = cudaMallocAsync((void**)&p, n * sizeof(T), stream);
        if (e != cudaSuccess) {
            p = nullptr;
            set_error("cudaMallocAsync(%zu bytes) failed: %s", n * sizeof(T), cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? VS_E_OOM : VS_E_CUDA;
        }
        return VS_OK;
    }
    void release() {
        if (p) cudaFreeAsync(p, s);
        p = nullptr;
    }
    T* release_ownership() {
        T* q = p;
        p = nullptr;
        return q;
    }
    ~Scratch() { release(); }
};

// Index memory, stream-ordered from the context's index pool (a cudaMalloc
// costs about 180 us here and a cudaFree 130 us; an index is some 25 of each).
// The stream has been waited for when the build returns.
template <class T>
int dalloc(T** p, size_t n, int64_t& bytes, vs_context* ctx) {
    if (n == 0) n = 1;
    const cudaError_t e = ctx->index_pool ? cudaMallocFromPoolAsync((void**)p, n * sizeof(T), ctx->index_pool, ctx->stream)
                                          : cudaMallocAsync((void**)p, n * sizeof(T), ctx->stream);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        set_error("allocation of %zu bytes of index memory failed: %s", n * sizeof(T), cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? VS_E_OOM : VS_E_CUDA;
    }
    bytes += (int64_t)(n * sizeof(T));
    return VS_OK;
}
// Return index memory no work uses any more to the pool.
inline void index_free(void* p) {
    if (p) cudaFreeAsync(p, cudaStreamLegacy);
}

// out[i] = sum(in[0..i)), n items; in == out allowed.  If d_total is non-null
// it receives sum(in[0..n)).
int exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* d_total, cudaStream_t s);
int exclusive_scan_u64(const uint64_t* in, uint64_t* out, int64_t n, uint64_t* d_total, cudaStream_t s);

// Stable LSD radix sort of (key, value) pairs by key bits [begin_bit,
// key_bits) (8 bits per pass).  Sorted data ends in keys / vals.
int radix_sort_u64_u32(uint64_t* keys, uint32_t* vals, int64_t n, int key_bits, cudaStream_t s, int begin_bit = 0);
int radix_sort_u32_u32(uint32_t* keys, uint32_t* vals, int64_t n, int key_bits, cudaStream_t s, int begin_bit = 0);
// The same for (left, right) pairs in place, by left then right: rows below
// 2^left_bits and 2^right_bits (at most 32 each; digits that are the same in
// every pair cost no pass).  by_runs: where left rows have few pairs each
// (n_left rows; 0: not known) only left is sorted by digits and equal left
// rows are ordered in their runs; bit 2 of *too_long (device memory) then
// reports a run too long for that, whose pairs are in left's order only.
int radix_sort_pairs(int32_t* left, int32_t* right, int64_t n, int left_bits, int right_bits, int64_t n_left,
                     bool by_runs, cudaStream_t s, unsigned long long* too_long);

}  // namespace vs
