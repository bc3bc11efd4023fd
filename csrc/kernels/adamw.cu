/**
 * One step of AdamW (Loshchilov and Hutter, "Decoupled Weight Decay Regularization", algorithm 2) on a flat slice: the update
 * between the reduce-scatter and the all-gather of dccl_b200/parallel/zero.py. Masters and moments are fp32; the gradient
 * arrives and the updated parameters leave in the parameters' own type.
 */
#include "adamw.hpp"
#include "launch_early.cuh"
#include "../device/reduce_ops.cuh"
#include <cstdint>
#include <cstdio>

namespace dccl {

struct AdamWArgs {
    float *master, *master_grad, *m, *v;
    const void* grad;
    void* out;
    size_t n;
    float decay;        // 1 - lr * weight_decay
    float w1;           // 1 - beta1
    float b2, w2;       // beta2, 1 - beta2
    float step;         // lr / (1 - beta1^t)
    float bc2_sqrt;     // sqrt(1 - beta2^t)
    float eps;
};
static_assert(launch_is_cheap(sizeof(AdamWArgs) + sizeof(bool)), "parameters of k_adamw");

/** N elements moved by one access. */
template <typename T, int N> struct alignas(sizeof(T) * N) Pack { T e[N]; };

constexpr int kAdamWThreads = 128;
constexpr int kAdamWN = 4;              // elements of one access: 16 bytes of fp32

/** Each operation rounds as torch's AdamW does one by one (moments as lerp and addcmul, true division and square root),
 *  except that a product feeding a sum is fused. The square of the gradient comes first, so that it overflows where torch's
 *  does: the element is then not updated any more. */
__device__ __forceinline__ void adamw_element(const AdamWArgs& a, float g, float& p, float& m, float& v) {
    p *= a.decay;
    m = a.w1 < 0.5f ? fmaf(a.w1, g - m, m) : fmaf(-(1.0f - a.w1), g - m, g);
    v = fmaf(a.w2, g * g, a.b2 * v);
    p = fmaf(-a.step, m / (sqrtf(v) / a.bc2_sqrt + a.eps), p);
}

/**
 * 32 bytes per 16-bit parameter (gradient in, its fp32 copy out, master and moments both ways, parameter out), no reuse:
 * HBM bounds it. One pass instead of the fourteen of the elementwise form, which reads and writes every fp32 array three to
 * six times: 44 M bf16 parameters take 209 us instead of 991 us (6.7 TB/s). One 16-byte access of each
 * fp32 array per thread and CTAs of 128; two accesses and CTAs of 256 took 0.3 % longer at 44 M and 1.7 % longer at 4 M
 * parameters (128 to 1024 threads with one, two and four accesses were tried). The arithmetic (two divisions, one square
 * root) hides behind the loads.
 */
template <typename T>
__global__ void __launch_bounds__(kAdamWThreads) k_adamw(const __grid_constant__ AdamWArgs a, bool vec) {
    wait_for_stream();
    using F = Pack<float, kAdamWN>;
    using P = Pack<T, kAdamWN>;
    const T* grad = reinterpret_cast<const T*>(a.grad);
    T* out = reinterpret_cast<T*>(a.out);
    if (vec) {
        const size_t i = (size_t)blockIdx.x * kAdamWThreads + threadIdx.x;
        if (i < a.n / kAdamWN) {
            const P g = reinterpret_cast<const P*>(grad)[i];
            F p = reinterpret_cast<const F*>(a.master)[i], m = reinterpret_cast<const F*>(a.m)[i], v = reinterpret_cast<const F*>(a.v)[i], gf;
            P o;
#pragma unroll
            for (int e = 0; e < kAdamWN; e++) {
                gf.e[e] = Traits<T>::up(g.e[e]);
                adamw_element(a, gf.e[e], p.e[e], m.e[e], v.e[e]);
                o.e[e] = Traits<T>::down(p.e[e]);
            }
            reinterpret_cast<F*>(a.master_grad)[i] = gf;
            reinterpret_cast<F*>(a.master)[i] = p;
            reinterpret_cast<F*>(a.m)[i] = m;
            reinterpret_cast<F*>(a.v)[i] = v;
            reinterpret_cast<P*>(out)[i] = o;
        }
    }
    // arrays that are not aligned, or the last elements of an odd length
    for (size_t i = (vec ? a.n / kAdamWN * kAdamWN : 0) + (size_t)blockIdx.x * kAdamWThreads + threadIdx.x; i < a.n; i += (size_t)gridDim.x * kAdamWThreads) {
        const float g = Traits<T>::up(grad[i]);
        a.master_grad[i] = g;
        adamw_element(a, g, a.master[i], a.m[i], a.v[i]);
        out[i] = Traits<T>::down(a.master[i]);
    }
}

} // namespace dccl

using namespace dccl;

extern "C" int dccl_adamw_flat(int device, int dtype, size_t n, void* master, void* master_grad, void* m, void* v, const void* grad, void* out,
                               double decay, double w1, double b2, double w2, double step, double bc2_sqrt, double eps, void* stream_v) {
    if (!n) return 0;
    AdamWArgs a = {(float*)master, (float*)master_grad, (float*)m, (float*)v, grad, out, n,
                   (float)decay, (float)w1, (float)b2, (float)w2, (float)step, (float)bc2_sqrt, (float)eps};
    const uintptr_t low = (uintptr_t)master | (uintptr_t)master_grad | (uintptr_t)m | (uintptr_t)v;
    const uintptr_t half = (uintptr_t)grad | (uintptr_t)out;
    const bool vec = low % 16 == 0 && half % (dtype == 7 ? 16 : 8) == 0;
    const size_t per = (size_t)kAdamWThreads * kAdamWN;
    const unsigned grid = (unsigned)((n + per - 1) / per);      // enough for 10^12 elements
    int prev = -1;
    cudaGetDevice(&prev);
    cudaError_t e = prev != device ? cudaSetDevice(device) : cudaSuccess;
    cudaStream_t stream = (cudaStream_t)stream_v;
    if (e == cudaSuccess)
        e = dtype == 6 ? launch_early(k_adamw<__half>, grid, kAdamWThreads, stream, a, vec) : dtype == 7 ? launch_early(k_adamw<float>, grid, kAdamWThreads, stream, a, vec)
            : dtype == 9 ? launch_early(k_adamw<__nv_bfloat16>, grid, kAdamWThreads, stream, a, vec) : cudaErrorInvalidValue;
    if (prev != device && prev >= 0) cudaSetDevice(prev);
    if (e == cudaSuccess) return 0;
    fprintf(stderr, "dccl_adamw_flat: %s\n", cudaGetErrorString(e));
    cudaGetLastError();
    return -1;
}
