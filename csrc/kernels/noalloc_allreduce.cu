/**
 * Implementation of dccl_allreduce_one_device_noalloc (see noalloc_allreduce.h).
 *
 * All ranks' buffers are on this device, so nothing has to travel between them: one pass reads every rank's element,
 * folds and writes the result to every rank. A thread owns its elements in ALL buffers, which is what makes in-place
 * calls (and outputs that are another rank's input) correct without any ordering between threads.
 */
#include "noalloc_allreduce.h"
#include "packed_ops.cuh"
#include "launch_early.cuh"
#include "../device/reduce_ops.cuh"
#include <cstdint>
#include <cstdio>

namespace dccl {

constexpr int kNoAllocThreads = 128;

/** 160 bytes; see launch_is_cheap. */
struct NoAllocArgs {
    int nranks;
    int op;
    unsigned count;        // elements per rank (at most DCCL_NOALLOC_MAX_BYTES of one-byte elements)
    unsigned per;          // elements per shard: shard j's fold starts at rank j
    unsigned head;         // elements before the first 16-byte boundary, the same in every buffer
    unsigned nvec;         // 16-byte vectors after it; 0: every element on its own
    const void* in[DCCL_NOALLOC_MAX_RANKS];
    void* out[DCCL_NOALLOC_MAX_RANKS];
    int* user_status;
};

/**
 * The last step of an element: ncclAvg scales. One-byte integers divide by a multiplication: |acc| <= 255 and at most 8
 * ranks, so |acc| * inv is less than 255 * 7 / 65536 < 1 / 8 of a unit above the quotient and its whole part is exact.
 * (8 x 256 KB of int8: 5.1 us of kernel for the average with sixteen divisions in a row and sums one by one, 2.5 us with
 * this and sums four at a time.)
 */
template <typename T, typename A> __device__ __forceinline__ T noalloc_finish(const NoAllocArgs& a, A acc) {
    if (a.op != 4) return Traits<T>::down(acc);
    if constexpr (sizeof(T) == 1) {
        const unsigned inv = 65535u / (unsigned)a.nranks + 1;      // ceil(65536 / nranks)
        const int q = (int)((unsigned)(acc < 0 ? -(int)acc : (int)acc) * inv >> 16);
        return (T)(acc < 0 ? -q : q);
    } else return Traits<T>::down(avg_finish<A>(acc, a.nranks));
}

/** Source number k of the fold of shard j: rank j, then the other ranks in ascending order. */
__device__ __forceinline__ int noalloc_source(int k, int j) { return k == 0 ? j : k - (k <= j ? 1 : 0); }

template <typename T, int OP>
__device__ __forceinline__ void noalloc_element(const NoAllocArgs& a, unsigned i) {
    using A = typename Traits<T>::Acc;
    const int n = a.nranks, j = (int)(i / a.per);
    T first = reinterpret_cast<const T*>(a.in[j])[i];
    if (n > 1) {
        A acc = Traits<T>::up(first);
        for (int k = 1; k < n; k++) acc = op_apply<OP, A>(acc, Traits<T>::up(reinterpret_cast<const T*>(a.in[noalloc_source(k, j)])[i]));
        first = noalloc_finish<T, A>(a, acc);
    }
    for (int p = 0; p < n; p++) reinterpret_cast<T*>(a.out[p])[i] = first;
}

/**
 * At most 4 MB move, so latency bounds this kernel: one 16-byte vector per thread with all ranks' loads in flight at
 * once, small CTAs so that the largest call (16384 vectors) still spreads over 128 SMs, one wave. The two-shot form it
 * replaced (shards pushed through a scratch array, two flag barriers between 4 CTAs per rank, ten memsets and a
 * cooperative launch) took 38.0 us a call for 8 x 1 KB and 43.2 us for 8 x 256 KB fp32 where this one takes 3.5 us, which is
 * the host's cost of a launch. Buffers at unequal distances from a 16-byte boundary go element by element, which stays behind
 * that launch, too: 8 x 256 KB take 3.9 us as bytes (before: 109 us) and 3.5 us as wider types (50 to 93 us).
 */
template <typename T, int OP>
__global__ void __launch_bounds__(kNoAllocThreads) k_noalloc_allreduce(const __grid_constant__ NoAllocArgs a) {
    using A = typename Traits<T>::Acc;
    constexpr int N = Vec16<T>::N;
    wait_for_stream();
    const unsigned t = blockIdx.x * kNoAllocThreads + threadIdx.x;
    const int n = a.nranks;
    if (t == 0 && a.user_status) *a.user_status = 0;
    if (t < a.nvec) {
        const unsigned i = a.head + t * N;
        const int j = (int)(i / a.per);
        if (n > 1 && j != (int)((i + N - 1) / a.per)) {      // a shard ends inside the vector (unaligned buffers only)
            for (int e = 0; e < N; e++) noalloc_element<T, OP>(a, i + e);
            return;
        }
        Vec16<T> v[DCCL_NOALLOC_MAX_RANKS];
#pragma unroll
        for (int k = 0; k < DCCL_NOALLOC_MAX_RANKS; k++)
            if (k < n) v[k] = ld_vec<T>(reinterpret_cast<const T*>(a.in[noalloc_source(k, j)]) + i);
        if (n > 1) {
            A acc[N];
            if constexpr (kFoldsBytes<T, OP>) {
#pragma unroll
                for (int k = 1; k < DCCL_NOALLOC_MAX_RANKS; k++) if (k < n) fold_packed<T, OP>(v[0], v[k]);
            }
#pragma unroll
            for (int e = 0; e < N; e++) acc[e] = Traits<T>::up(v[0].e[e]);
            if constexpr (!kFoldsBytes<T, OP>) {
#pragma unroll
                for (int k = 1; k < DCCL_NOALLOC_MAX_RANKS; k++) {
                    if (k < n) {
#pragma unroll
                        for (int e = 0; e < N; e++) acc[e] = op_apply<OP, A>(acc[e], Traits<T>::up(v[k].e[e]));
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < N; e++) v[0].e[e] = noalloc_finish<T, A>(a, acc[e]);
        }
#pragma unroll
        for (int p = 0; p < DCCL_NOALLOC_MAX_RANKS; p++)
            if (p < n) st_vec<T>(reinterpret_cast<T*>(a.out[p]) + i, v[0]);
        return;
    }
    // the elements outside the vectors: before the first boundary, then after the last one
    unsigned i = t - a.nvec;
    if (i >= a.head) i += a.nvec * N;
    if (i < a.count) noalloc_element<T, OP>(a, i);
}

static_assert(launch_is_cheap(sizeof(NoAllocArgs)), "parameters of k_noalloc_allreduce");

} // namespace dccl

using namespace dccl;

extern "C" int dccl_allreduce_one_device_noalloc(int nranks, int dtype, int op, size_t count, const void* const* inputs,
                                                 void* const* outputs, int* device_status, void* stream_v) {
    cudaStream_t stream = (cudaStream_t)stream_v;
    if (nranks < 1 || nranks > DCCL_NOALLOC_MAX_RANKS || dtype < 0 || dtype > 9 || op < 0 || op > 4 || !inputs || !outputs) {
        fprintf(stderr, "dccl_allreduce_one_device_noalloc: bad argument (nranks %d, dtype %d, op %d)\n", nranks, dtype, op);
        return DCCL_NOALLOC_BAD_ARGUMENT;
    }
    static const size_t kSizes[10] = {1, 1, 4, 4, 8, 8, 2, 4, 8, 2};
    size_t es = kSizes[dtype];
    if (count > DCCL_NOALLOC_MAX_BYTES / es) {
        fprintf(stderr, "dccl_allreduce_one_device_noalloc: %zu elements of %zu bytes per rank are above the limit of %u bytes of this entry point\n",
                count, es, (unsigned)DCCL_NOALLOC_MAX_BYTES);
        return DCCL_NOALLOC_TOO_LARGE;
    }
    for (int r = 0; r < nranks; r++)
        if (count && (!inputs[r] || !outputs[r])) {
            fprintf(stderr, "dccl_allreduce_one_device_noalloc: null buffer for rank %d\n", r);
            return DCCL_NOALLOC_BAD_ARGUMENT;
        }
    if (count == 0) return DCCL_NOALLOC_OK;
    // one rank's result is a copy of its input, which no pointer is too odd for: between two elements it goes by bytes
    if (nranks == 1 && ((uintptr_t)inputs[0] | (uintptr_t)outputs[0]) % es != 0) {
        count *= es;
        dtype = 1;
        es = 1;
    }
    // everywhere else the kernel loads and stores elements
    for (int r = 0; r < nranks; r++)
        if ((((uintptr_t)inputs[r] | (uintptr_t)outputs[r]) & (es - 1)) != 0) {
            fprintf(stderr, "dccl_allreduce_one_device_noalloc: buffer of rank %d lies between two elements of %zu bytes\n", r, es);
            return DCCL_NOALLOC_BAD_ARGUMENT;
        }

    NoAllocArgs a;
    a.nranks = nranks;
    a.op = op;
    a.count = (unsigned)count;
    // shards as the two-shot all-reduce cuts them: whole 16-byte vectors
    const unsigned ve = (unsigned)(16 / es);
    a.per = (unsigned)((count + nranks - 1) / nranks + ve - 1) / ve * ve;
    // 16-byte accesses when every buffer has the same distance to a 16-byte boundary
    const uintptr_t mis = (uintptr_t)inputs[0] & 15u;
    bool vec = true;
    for (int r = 0; r < DCCL_NOALLOC_MAX_RANKS; r++) {
        a.in[r] = r < nranks ? inputs[r] : nullptr;
        a.out[r] = r < nranks ? outputs[r] : nullptr;
        if (r < nranks) vec = vec && ((uintptr_t)inputs[r] & 15u) == mis && ((uintptr_t)outputs[r] & 15u) == mis;
    }
    a.head = vec ? (unsigned)((16 - mis) % 16 / es) : 0;
    if (a.head > a.count) a.head = a.count;
    a.nvec = vec ? (a.count - a.head) / ve : 0;
    a.user_status = device_status;
    const unsigned threads = a.nvec + (a.count - a.nvec * ve);
    const unsigned grid = (threads + kNoAllocThreads - 1) / kNoAllocThreads;
    cudaError_t e = cudaErrorInvalidValue;
#define CALL(T, OP) e = launch_early(k_noalloc_allreduce<T, OP>, grid, kNoAllocThreads, stream, a)
    DCCL_DISPATCH_TYPE_OP(dtype, op, CALL)
#undef CALL
    if (e != cudaSuccess) {
        fprintf(stderr, "dccl_allreduce_one_device_noalloc: launch: %s\n", cudaGetErrorString(e));
        cudaGetLastError();
        return DCCL_NOALLOC_CUDA_ERROR;
    }
    return DCCL_NOALLOC_OK;
}
