/**
 * All-reduce among buffers that live on ONE device, through an entry point that
 * allocates nothing.
 *
 * This entry point has no counterpart in the original DCCL; it exists for
 * callers of this library that are not allowed to allocate device memory at
 * the moment they need a reduction:
 *
 *   - code that runs while the device memory is fully handed out to a
 *     framework's caching allocator or to a serving engine's KV-cache pool, so
 *     that a cudaMalloc may fail or stall (it synchronises the whole device);
 *   - code on a latency-critical path (one process driving several model
 *     replicas or pipeline partitions on one GPU, "threads as ranks") where
 *     the implicit device-wide synchronisation of cudaMalloc / cudaFree is not
 *     acceptable;
 *   - health checks that must work in a process whose memory budget is spent.
 *
 * The communicator-based API creates a pool per communicator (cuMemCreate /
 * cudaMalloc at init) and the test harness dccl_emu_collective allocates the
 * pools of its virtual ranks on every call. This entry point needs no scratch
 * at all: the buffers are on one device, so one kernel reads every rank's
 * element, folds and writes the result to every rank.
 *
 * What it computes: for r in [0, nranks): outputs[r][i] = op(inputs[0][i], ...,
 * inputs[nranks-1][i]), i in [0, count). Same accumulation order as the
 * two-shot variant of ncclAllReduce: the vector is cut into nranks shards of
 * whole 16-byte vectors, and the fold of shard j starts at rank j and goes on
 * with the other ranks in ascending order.
 *
 * Limits and rules:
 *   - nranks 1..DCCL_NOALLOC_MAX_RANKS, count * element size <=
 *     DCCL_NOALLOC_MAX_BYTES per rank; larger requests are refused with
 *     DCCL_NOALLOC_TOO_LARGE and a message on stderr, nothing is launched.
 *   - One ordinary kernel launch on `stream`, no state between calls: calls on
 *     different streams may overlap, and a call can be captured in a graph.
 *   - inputs / outputs are host arrays of nranks device pointers (read during
 *     the call, not kept). Element pointers must be aligned to the element
 *     size, or the call is refused with DCCL_NOALLOC_BAD_ARGUMENT (with one
 *     rank, whose call is a copy, they need not be); buffers that all have the
 *     same distance to a 16-byte boundary take the vector path. outputs[r] may
 *     equal inputs[r] (or another rank's input); buffers that overlap only
 *     partly are not supported.
 *   - device_status, when not null, is a device int the kernel sets to 0. (The
 *     ranks no longer wait for one another, so there is no wait that could give
 *     up.)
 *   - No cudaMalloc, cudaFree, cudaMallocAsync, cudaHostAlloc or allocating
 *     library routine is called, on any path.
 */
#pragma once
#include <stddef.h>

#ifdef __cplusplus
extern "C" {
#endif

#define DCCL_NOALLOC_MAX_RANKS 8
#define DCCL_NOALLOC_MAX_BYTES (256u * 1024u)
/* device memory the library holds for this entry point, for one rank and altogether: none */
#define DCCL_NOALLOC_RANK_BYTES 0u
#define DCCL_NOALLOC_SCRATCH_BYTES 0u

#define DCCL_NOALLOC_OK 0
#define DCCL_NOALLOC_BAD_ARGUMENT (-1)
#define DCCL_NOALLOC_TOO_LARGE (-2)
#define DCCL_NOALLOC_CUDA_ERROR (-3)

/**
 * dtype: ncclDataType_t value (0 int8 ... 9 bfloat16); op: ncclRedOp_t value (0 sum, 1 prod, 2 max,
 * 3 min, 4 avg); stream: a cudaStream_t (0 for the default stream). Returns DCCL_NOALLOC_OK when the
 * work was enqueued, or one of the negative codes above after printing the reason to stderr.
 */
int dccl_allreduce_one_device_noalloc(int nranks, int dtype, int op, size_t count, const void* const* inputs,
                                      void* const* outputs, int* device_status, void* stream);

#ifdef __cplusplus
}
#endif
