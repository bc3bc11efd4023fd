/**
 * Single-GPU kernels: copy, pairwise reduce (the operation of the original's
 * only kernel, reference src/core/reduce.cu:9-38, as a vectorised, operator-
 * templated grid), and the bounded-wait self test.
 */
#include "kernels.hpp"
#include "../device/reduce_ops.cuh"

namespace dccl {

static int g_sm_count = 0;
static int sm_count() {
    if (!g_sm_count) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        g_sm_count = n > 0 ? n : 148;
    }
    return g_sm_count;
}

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

/** The 16 bytes at `p`, which lies k bytes behind a 16-byte boundary: one aligned vector, or a window over two. */
__device__ __forceinline__ uint4 load16(const char* p, unsigned k) {
    const uint4* q = reinterpret_cast<const uint4*>(p - k);
    const uint4 a = q[0];
    return k == 0 ? a : window16(a, q[1], k);
}

/**
 * How a range is cut so that every store is a whole, aligned 16-byte vector whatever the two pointers are: `head` bytes up
 * to the destination's first boundary, `nv` vectors, the rest. The source then lies `shift` bytes behind a boundary for all
 * vectors alike. A source vector is read through the two aligned ones it lies in, so with a shift one vector more goes to
 * the head where its first aligned one would begin before the source, and to the rest where its second one would end
 * behind it: nothing outside the buffers is read.
 */
struct Cut {
    size_t head, nv, rest;
    unsigned shift;
};

static Cut cut_range(const void* dst, const void* src, size_t bytes) {
    Cut c;
    c.head = (16 - (reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u;
    c.shift = (unsigned)((reinterpret_cast<uintptr_t>(src) + c.head) & 15u);
    if (c.head < c.shift) c.head += 16;
    if (c.head > bytes) c.head = bytes;
    c.nv = (bytes - c.head + c.shift) / 16;
    if (c.shift && c.nv) c.nv--;
    c.rest = bytes - c.head - c.nv * 16;
    return c;
}

/**
 * HBM bounds a large copy, launch and latency a small one. Every thread moves two vectors and the CTAs follow each other
 * through memory, so that all SMs work in one window of a few MB: 1 GiB takes 312 us (6.9 TB/s of reads and writes) where
 * two resident CTAs per SM, each on a contiguous piece of its own, took 363 us (296 places of memory open at once). The
 * same shape is within 1 % of the best from 64 KB to 1 GiB (one to four vectors, 256 to 1024 threads, 16- and 32-byte
 * accesses were tried), so there is one. Pointers with different distances to a 16-byte boundary cost a second load, which
 * the L1 cache serves, and a few selects: 26 MB of bf16 from a source 6 bytes off take 12.3 us where a loop over single bytes
 * took 88.2 us.
 */
constexpr int kCopyThreads = 256, kCopyU = 2;
__global__ void __launch_bounds__(kCopyThreads) k_local_copy(char* __restrict__ dst, const char* __restrict__ src, const __grid_constant__ Cut c) {
    const size_t i0 = (size_t)blockIdx.x * (kCopyThreads * kCopyU) + threadIdx.x;
    uint4 v[kCopyU];
#pragma unroll
    for (int u = 0; u < kCopyU; u++)
        if (i0 + u * kCopyThreads < c.nv) v[u] = load16(src + c.head + (i0 + u * kCopyThreads) * 16, c.shift);
#pragma unroll
    for (int u = 0; u < kCopyU; u++)
        if (i0 + u * kCopyThreads < c.nv) *reinterpret_cast<uint4*>(dst + c.head + (i0 + u * kCopyThreads) * 16) = v[u];
    if (blockIdx.x == 0) {      // at most 31 bytes before and 47 behind the vectors
        for (size_t j = threadIdx.x; j < c.head; j += kCopyThreads) dst[j] = src[j];
        for (size_t j = c.head + c.nv * 16 + threadIdx.x; j < c.head + c.nv * 16 + c.rest; j += kCopyThreads) dst[j] = src[j];
    }
}

/**
 * acc[i] = op(acc[i], in[i]). Three streams of HBM traffic and nothing else, so what matters is bytes in flight:
 * every thread keeps kLocalU 16-byte vectors of each operand outstanding (128 KB per SM with two resident CTAs),
 * each CTA on one contiguous piece.
 */
constexpr int kLocalU = 4;
template <typename T, int OP>
__global__ void __launch_bounds__(512) k_local_reduce(T* acc, const T* __restrict__ in, size_t count, int avg) {
    using A = typename Traits<T>::Acc;
    constexpr size_t VE = 16 / sizeof(T);
    constexpr int N = Vec16<T>::N;
    const size_t per = ((count + gridDim.x - 1) / gridDim.x + VE - 1) / VE * VE;
    const size_t lo = per * blockIdx.x;
    if (lo >= count) return;
    const size_t n = count - lo < per ? count - lo : per;
    T* a = acc + lo;
    const T* b = in + lo;
    size_t done = 0;
    if (aligned16(a) && aligned16(b)) {
        const size_t nv = n / N, tid = threadIdx.x, nt = blockDim.x;
        size_t i = tid;
        for (; i + (size_t)(kLocalU - 1) * nt < nv; i += (size_t)kLocalU * nt) {
            Vec16<T> x[kLocalU], y[kLocalU];
#pragma unroll
            for (int u = 0; u < kLocalU; u++) { x[u] = ld_vec<T>(a + (i + (size_t)u * nt) * N); y[u] = ld_vec<T>(b + (i + (size_t)u * nt) * N); }
#pragma unroll
            for (int u = 0; u < kLocalU; u++) {
#pragma unroll
                for (int e = 0; e < N; e++) x[u].e[e] = Traits<T>::down(op_apply<OP, A>(Traits<T>::up(x[u].e[e]), Traits<T>::up(y[u].e[e])));
                st_vec<T>(a + (i + (size_t)u * nt) * N, x[u]);
            }
        }
        for (; i < nv; i += nt) {
            Vec16<T> x = ld_vec<T>(a + i * N), y = ld_vec<T>(b + i * N);
#pragma unroll
            for (int e = 0; e < N; e++) x.e[e] = Traits<T>::down(op_apply<OP, A>(Traits<T>::up(x.e[e]), Traits<T>::up(y.e[e])));
            st_vec<T>(a + i * N, x);
        }
        done = nv * N;
    }
    // ragged end, or operands that are not 16-byte aligned
    const T* ins[1] = {b + done};
    if (n > done) reduce_range<T, OP>(a + done, nullptr, a + done, ins, 1, n - done, avg != 0, 2);
}

cudaError_t launch_local_copy(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    if (!bytes || dst == src) return cudaSuccess;
    const Cut c = cut_range(dst, src, bytes);
    const size_t per = (size_t)kCopyThreads * kCopyU, grid = (c.nv + per - 1) / per;
    k_local_copy<<<(unsigned)(grid ? grid : 1), kCopyThreads, 0, stream>>>((char*)dst, (const char*)src, c);
    return cudaGetLastError();
}

cudaError_t launch_local_reduce(void* acc, const void* in, size_t count, ncclDataType_t dt, ncclRedOp_t op, cudaStream_t stream) {
    if (!count) return cudaSuccess;
    const size_t es = dt == ncclInt8 || dt == ncclUint8 ? 1 : dt == ncclFloat16 || dt == ncclBfloat16 ? 2
                      : dt == ncclInt32 || dt == ncclUint32 || dt == ncclFloat32 ? 4 : 8;
    size_t want = (count * es + (64u << 10) - 1) / (64u << 10);
    int grid = (int)(want < (size_t)(2 * sm_count()) ? want : (size_t)(2 * sm_count()));   // two resident CTAs per SM: one wave
    if (grid < 1) grid = 1;
    const int avg = 0;   // a pairwise fold has no world size: ncclAvg accumulates like ncclSum here
#define CALL(T, OP) k_local_reduce<T, OP><<<grid, 512, 0, stream>>>((T*)acc, (const T*)in, count, avg)
    DCCL_DISPATCH_TYPE_OP((int)dt, (int)op, CALL)
#undef CALL
    return cudaGetLastError();
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
