/**
 * The two ends of an early launch, for tests of the kernels that are launched so: a kernel that lets the launch after it
 * start at once and writes much later, and one that tells when it was started.
 */
#include "../kernels/launch_early.cuh"
#include <cstdint>
#include <cstdio>

namespace {

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__global__ void k_early_producer(uint32_t* dst, const uint32_t* src, size_t words, unsigned spin_us, unsigned long long* end) {
    cudaTriggerProgrammaticLaunchCompletion();
    const unsigned long long t0 = now_ns();
    // bounded twice: by the clock, and by the number of naps
    for (unsigned i = 0; i < 4 * spin_us && now_ns() - t0 < 1000ull * spin_us; i++) __nanosleep(1000);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) dst[i] = src[i];
    if (end && blockIdx.x == 0 && threadIdx.x == 0) *end = now_ns();
}

__global__ void k_early_observer(unsigned long long* start) {
    if (threadIdx.x == 0) *start = now_ns();
    dccl::wait_for_stream();
}

int result(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return 0;
    fprintf(stderr, "dccl emulation: %s: %s\n", what, cudaGetErrorString(e));
    cudaGetLastError();
    return -1;
}

} // namespace

extern "C" {

/** dst[0..words) = src[0..words), written `spin_us` microseconds (at most 2000) after the launch behind this one was let go.
 *  end, when not null: the time of that, in nanoseconds of the device's clock. */
int dccl_emu_early_producer(void* dst, const void* src, size_t words, unsigned spin_us, void* end, void* stream) {
    if (spin_us > 2000) spin_us = 2000;
    k_early_producer<<<8, 256, 0, (cudaStream_t)stream>>>((uint32_t*)dst, (const uint32_t*)src, words, spin_us, (unsigned long long*)end);
    return result(cudaGetLastError(), "early producer");
}

/** Launched as the library's own kernels are: *start is the time at which it ran, before it waited. */
int dccl_emu_early_observer(void* start, void* stream) {
    return result(dccl::launch_early(k_early_observer, 1, 32, (cudaStream_t)stream, (unsigned long long*)start), "early observer");
}

} // extern "C"
