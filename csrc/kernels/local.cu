/**
 * Single-GPU kernels: copy, pairwise reduce (the operation of the original's
 * only kernel, reference src/core/reduce.cu:9-38, as a vectorised, operator-
 * templated grid), and the bounded-wait self test.
 */
#include "packed_ops.cuh"
#include "launch_early.cuh"
#include "kernels.hpp"
#include "local_shapes.hpp"
#include "../device/reduce_ops.cuh"

namespace dccl {

/** Bytes k .. k+15 of the 32 bytes (a, b); k is the same for all threads of a launch. */
__device__ __forceinline__ uint4 window16(uint4 a, uint4 b, unsigned k) {
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t x[6], y[5];
#pragma unroll
    for (int j = 0; j < 6; j++) x[j] = k & 8 ? w[j + 2] : w[j];
#pragma unroll
    for (int j = 0; j < 5; j++) y[j] = k & 4 ? x[j + 1] : x[j];
    const unsigned r = (k & 3) * 8;
    return make_uint4(__funnelshift_r(y[0], y[1], r), __funnelshift_r(y[1], y[2], r), __funnelshift_r(y[2], y[3], r), __funnelshift_r(y[3], y[4], r));
}

/** The 16 bytes k bytes behind the 16-byte boundary `q`: the aligned vector there, or a window over it and the next one. Two
 *  steps, so that a thread has all its loads in flight before it needs one: taken in one step per vector, the loads of the
 *  later vectors waited for the window of the first. Three sets of 26 MB copied from a source 6 bytes off: 10.05 -> 9.40 us. */
struct Window { uint4 a, b; };
__device__ __forceinline__ void load(Window& w, const void* q, unsigned k) {
    w.a = reinterpret_cast<const uint4*>(q)[0];
    if (k) w.b = reinterpret_cast<const uint4*>(q)[1];
}
__device__ __forceinline__ uint4 cut_out(const Window& w, unsigned k) { return k ? window16(w.a, w.b, k) : w.a; }

/**
 * How a range is cut so that every store is a whole, aligned 16-byte vector whatever the two pointers are: `head` bytes up
 * to the destination's first boundary, `nv` vectors, the rest. The source then lies `shift` bytes behind a boundary for all
 * vectors alike. A source vector is read through the two aligned ones it lies in, so with a shift one vector more goes to
 * the head where its first aligned one would begin before the source, and to the rest where its second one would end
 * behind it: nothing outside the buffers is read. The ends are bytes so that, with the two pointers, the parameters of the
 * kernels below are 32 bytes: with 48, the fold of 1 MiB took 3.69 us a call instead of 3.32, and a one-rank all-reduce of 4 KB
 * 5.56 instead of 5.21.
 */
struct Cut {
    size_t nv;
    uint8_t head, shift, rest;
};
static_assert(launch_is_cheap(2 * sizeof(void*) + sizeof(Cut)), "parameters of k_local_copy and k_local_reduce");

static Cut cut_range(const void* dst, const void* src, size_t bytes) {
    size_t head = (16 - (reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u;
    const size_t shift = (reinterpret_cast<uintptr_t>(src) + head) & 15u;
    if (head < shift) head += 16;
    if (head > bytes) head = bytes;
    size_t nv = (bytes - head + shift) / 16;
    if (shift && nv) nv--;
    return {nv, (uint8_t)head, (uint8_t)shift, (uint8_t)(bytes - head - nv * 16)};      // neither end is longer than 30 bytes
}

/**
 * HBM bounds a large copy, launch and latency a small one. Every thread moves two vectors and the CTAs follow each other
 * through memory, so that all SMs work in one window of a few MB: 1 GiB takes 305 us (7.0 TB/s of reads and writes) where
 * two resident CTAs per SM, each on a contiguous piece of its own, took 363 us (296 places of memory open at once). Pointers
 * with different distances to a 16-byte boundary cost a second load, which the L1 cache serves, and a few selects: 26 MB of
 * bf16 from a source 6 bytes off take 9.4 us where a loop over single bytes took 88.2 us.
 */
constexpr int kCopyU = 2;
template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_local_copy(char* dst, const char* src, const __grid_constant__ Cut c) {
    wait_for_stream();
    const size_t i0 = (size_t)blockIdx.x * (THREADS * kCopyU) + threadIdx.x;
    const char* q = src + c.head - c.shift;
    Window w[kCopyU];
#pragma unroll
    for (int u = 0; u < kCopyU; u++)
        if (i0 + u * THREADS < c.nv) load(w[u], q + (i0 + u * THREADS) * 16, c.shift);
#pragma unroll
    for (int u = 0; u < kCopyU; u++)
        if (i0 + u * THREADS < c.nv) *reinterpret_cast<uint4*>(dst + c.head + (i0 + u * THREADS) * 16) = cut_out(w[u], c.shift);
    if (blockIdx.x == 0) {      // at most 30 bytes before and 30 behind the vectors
        for (size_t j = threadIdx.x; j < c.head; j += THREADS) dst[j] = src[j];
        for (size_t j = c.head + c.nv * 16 + threadIdx.x; j < c.head + c.nv * 16 + c.rest; j += THREADS) dst[j] = src[j];
    }
}

/**
 * acc[i] = op(acc[i], in[i]): three streams of HBM traffic and nothing else, the CTAs following each other through memory as in
 * the copy: 1 GiB fp32 takes 448 us (7.2 TB/s), 25 MiB bf16 12.7 us and 1 MiB 3.3 us (the host's cost of the call), where two
 * resident CTAs per SM with eight vectors in flight per thread, each CTA on a piece of at least 64 KB, took 520, 16.4 and 5.1 us.
 * Operands at different distances from a 16-byte boundary read `in` through a window as the copy does: 12 MB of fp16 24.6 ->
 * 3.9 us (before: one element per access). The elements outside the vectors get threads of their own behind the vectors' threads.
 */
template <typename T, int OP, int THREADS, int U>
__global__ void __launch_bounds__(THREADS) k_local_reduce(T* acc, const T* in, const __grid_constant__ Cut c) {
    using A = typename Traits<T>::Acc;
    constexpr int N = Vec16<T>::N;
    wait_for_stream();
    const size_t t0 = (size_t)blockIdx.x * (THREADS * U) + threadIdx.x;
    const size_t head = c.head / sizeof(T);
    T* p = acc + head;
    const char* q = reinterpret_cast<const char*>(in + head) - c.shift;
    Window w[U];
    Vec16<T> x[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const size_t t = t0 + u * THREADS;
        if (t >= c.nv) continue;
        load(w[u], q + t * 16, c.shift);
        x[u] = ld_vec<T>(p + t * N);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const size_t t = t0 + u * THREADS;
        if (t < c.nv) {
            Vec16<T> y;
            *reinterpret_cast<uint4*>(&y) = cut_out(w[u], c.shift);
            if constexpr (kFoldsBytes<T, OP> || kFoldsPairs<T, OP>) fold_packed<T, OP>(x[u], y);
            else {
#pragma unroll
                for (int e = 0; e < N; e++) x[u].e[e] = Traits<T>::down(op_apply<OP, A>(Traits<T>::up(x[u].e[e]), Traits<T>::up(y.e[e])));
            }
            st_vec<T>(p + t * N, x[u]);
            continue;
        }
        size_t i = t - c.nv;
        if (i >= head) i += c.nv * N;
        if (i < head + c.nv * N + c.rest / sizeof(T)) acc[i] = Traits<T>::down(op_apply<OP, A>(Traits<T>::up(acc[i]), Traits<T>::up(in[i])));
    }
}

cudaError_t launch_local_copy(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    if (!bytes || dst == src) return cudaSuccess;
    const Cut c = cut_range(dst, src, bytes);
    const unsigned threads = copy_threads(bytes);
    const size_t per = (size_t)threads * kCopyU, grid = (c.nv + per - 1) / per;
    return launch_early(threads == 1024 ? k_local_copy<1024> : k_local_copy<256>, (unsigned)(grid ? grid : 1), threads, stream, (char*)dst, (const char*)src, c);
}

cudaError_t launch_local_reduce(void* acc, const void* in, size_t count, ncclDataType_t dt, ncclRedOp_t op, cudaStream_t stream) {
    if (!count) return cudaSuccess;
    const size_t es = dt == ncclInt8 || dt == ncclUint8 ? 1 : dt == ncclFloat16 || dt == ncclBfloat16 ? 2
                      : dt == ncclInt32 || dt == ncclUint32 || dt == ncclFloat32 ? 4 : 8;
    if ((reinterpret_cast<uintptr_t>(acc) | reinterpret_cast<uintptr_t>(in)) % es) return cudaErrorInvalidValue;
    // a pairwise fold has no world size: ncclAvg accumulates like ncclSum here
    const Cut c = cut_range(acc, in, count * es);
    const size_t threads = c.nv + (c.head + c.rest) / es;
    cudaError_t e = cudaErrorInvalidValue;
#define SHAPED(T, OP, THREADS, U) launch_early(k_local_reduce<T, OP, THREADS, U>, (unsigned)((threads + THREADS * U - 1) / (THREADS * U)), THREADS, stream, (T*)acc, (const T*)in, c)
#define CALL(T, OP) e = two_vectors(count * es) ? SHAPED(T, OP, 128, 2) : SHAPED(T, OP, 512, 1)
    DCCL_DISPATCH_TYPE_OP((int)dt, (int)op, CALL)
#undef CALL
#undef SHAPED
    return e;
}

/** Waits for a flag value that nothing ever writes; must return through the timeout path. */
__global__ void k_wait_probe(const __grid_constant__ DevComm c) {
    if (threadIdx.x == 0) {
        uint32_t* slot = flag_slot(c.pool[c.rank], kMaxCtas - 1, kMaxPeers - 1);
        const uint32_t never = ld_volatile_u32(slot) + 0x40000000u;
        wait_flag_ge(c, slot, never, kMaxPeers - 1, 900, 0);
    }
}

cudaError_t launch_wait_probe(const DevComm& c, cudaStream_t stream) {
    void* params[] = {const_cast<DevComm*>(&c)};
    return cudaLaunchKernel((const void*)k_wait_probe, dim3(1), dim3(32), params, 0, stream);
}

} // namespace dccl
