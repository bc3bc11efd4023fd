"""Compile-time properties of the kernels' dispatch; a compiler is all these tests take."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKED = """
#include "csrc/kernels/packed_ops.cuh"
using namespace dccl;
struct OneByte { unsigned char b; };
template <typename T, int OP> constexpr bool alone() { return !kFoldsBytes<T, OP> && !kFoldsPairs<T, OP>; }
static_assert(alone<short, OP_SUM>() && alone<unsigned short, OP_MAX>() && alone<OneByte, OP_MIN>() && alone<float, OP_SUM>(), "types without packed operations");
static_assert(kFoldsPairs<__half, OP_SUM> && kFoldsPairs<__nv_bfloat16, OP_MAX> && kFoldsBytes<signed char, OP_SUM> && kFoldsBytes<unsigned char, OP_MIN>, "types with them");
static_assert(alone<__half, OP_PROD>() && alone<__nv_bfloat16, OP_PROD>() && alone<signed char, OP_PROD>(), "products");
"""


# Each type by its name (csrc/kernels/packed_ops.cuh): another type of the same size needs other instructions.
def test_types_that_fold_several_elements_at_a_time(tmp_path):
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    (tmp_path / "types.cu").write_text(PACKED)
    res = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + ROOT, "-I" + os.path.join(ROOT, "include"), "-DDCCL_WITH_CUDA_RUNTIME",
                          "-c", str(tmp_path / "types.cu"), "-o", str(tmp_path / "types.o")], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]


SHAPES = """
#include "csrc/kernels/local_shapes.hpp"
constexpr size_t kL2 = 126000000;
constexpr bool copies_out_of_l2_in_small_ctas() {
    for (size_t bytes = 4096; 2 * bytes <= kL2; bytes += 4096)
        if (dccl::copy_threads(bytes) != 256) return false;
    return true;
}
static_assert(copies_out_of_l2_in_small_ctas(), "a pair of buffers that fits into L2");
static_assert(dccl::copy_threads(kL2) == 1024 && dccl::copy_threads(size_t(1) << 30) == 1024 && dccl::copy_threads(size_t(1) << 40) == 1024, "a pair that does not");
"""


# A pair of buffers that fits into L2 is copied from there when it comes again, 6 to 12 % slower in CTAs of 1024.
def test_copies_that_can_come_out_of_l2_keep_their_shape(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("needs a C++ compiler")
    (tmp_path / "shapes.cpp").write_text(SHAPES)
    res = subprocess.run([cxx, "-std=c++17", "-fsyntax-only", "-fconstexpr-loop-limit=1000000", "-I" + ROOT, str(tmp_path / "shapes.cpp")], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
