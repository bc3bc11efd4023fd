/**
 * Entry point of the one-kernel AdamW update (adamw.cu), for its definition and for callers that find it by address.
 */
#pragma once
#include <cstddef>

/**
 * AdamW on `n` elements that live on `device`: master, moments and out are updated, master_grad receives the gradient in
 * fp32. dtype: ncclDataType_t of grad and out (float16, float32 or bfloat16). Returns 0, or -1 after a message on stderr.
 */
extern "C" int dccl_adamw_flat(int device, int dtype, size_t n, void* master, void* master_grad, void* m, void* v, const void* grad, void* out,
                               double decay, double w1, double b2, double w2, double step, double bc2_sqrt, double eps, void* stream);
