/**
 * Launches that are set up while the kernel before them in the stream drains (programmatic dependent launch), for the
 * kernels whose calls are short enough for the gap between two launches to count.
 */
#pragma once
#include <cuda_runtime.h>

namespace dccl {

/** First statement of such a kernel, before any access to memory, in every thread: the work before it in the stream is
 *  done and visible. (The kernels do not announce themselves early to the launch after them: whatever follows starts, as
 *  after any kernel, when they are done.) No pointer of such a kernel is __restrict__ and none is read by __ldg: either
 *  declares its memory unchanged from the kernel's start on, which lies before that work, and lets a load be taken before
 *  the wait. */
__device__ __forceinline__ void wait_for_stream() { cudaGridDependencySynchronize(); }

/**
 * What a launch costs the host depends on the size of the kernel's parameters, with a period of 64 bytes: 17 to 32 bytes past a
 * multiple of 64 took 1.54 us, every other size 1.81 to 1.94 us (8 to 320 bytes in steps of 8, calls back to back). A kernel
 * whose calls are short packs its parameters into such a size.
 */
constexpr bool launch_is_cheap(size_t parameter_bytes) { return parameter_bytes % 64 > 16 && parameter_bytes % 64 <= 32; }

/**
 * Measured on back-to-back calls: the pairwise fold of 25 MiB of bf16 14.35 -> 12.7 us, of 12 MB of unaligned fp16
 * 6.15 -> 4.4 us, the copy of 26 MB 12.3 -> 10.0 us; nothing at 1 GiB. A capturing stream gets an ordinary launch: the
 * edge a programmatic one leaves in a graph carries data that not every user of the capture API expects.
 */
template <typename... P, typename... A>
inline cudaError_t launch_early(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t stream, A... args) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess) cudaGetLastError();      // the launch reports it
    else if (capturing == cudaStreamCaptureStatusNone) { cfg.attrs = &attr; cfg.numAttrs = 1; }
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

} // namespace dccl
