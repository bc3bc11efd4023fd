"""What the one-GPU calls decide on the host, before anything reaches a GPU."""
import ctypes
import os
import subprocess

import pytest

from dccl_b200.comm import FLOAT32, FLOAT64, OPS

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def cuda_lib(dccl_lib):
    if not hasattr(dccl_lib, "dccl_allreduce_one_device_noalloc"):
        pytest.skip("library built without CUDA")
    return dccl_lib


@pytest.mark.parametrize("dtype,size", [(FLOAT32, 4), (FLOAT64, 8)])
@pytest.mark.parametrize("where", ["input", "output"])
def test_one_device_all_reduce_refuses_a_pointer_between_elements(cuda_lib, capfd, dtype, size, where):
    fn = cuda_lib.dccl_allreduce_one_device_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    good, odd = (ctypes.c_void_p * 2)(0x10000, 0x20000), (ctypes.c_void_p * 2)(0x10000, 0x20000 + size // 2)
    ins, outs = (odd, good) if where == "input" else (good, odd)
    assert fn(2, dtype, OPS["sum"], 4, ins, outs, None, None) == -1        # bad argument; the addresses are never used
    assert "rank 1" in capfd.readouterr().err
    assert fn(2, dtype, OPS["sum"], 0, ins, outs, None, None) == 0         # no element, nothing to refuse


def test_early_launched_kernels_promise_nothing_about_their_inputs():
    """A kernel that starts before the one ahead of it has written must not declare what it reads read-only for as long as it
    runs: such loads may be taken before the wait."""
    found = 0
    folder = os.path.join(ROOT, "csrc", "kernels")
    for name in sorted(os.listdir(folder)):
        text = open(os.path.join(folder, name)).read()
        for part in text.split("__global__")[1:]:
            signature, body = part.split("{", 1)
            body = body.split("\n}", 1)[0]
            if "wait_for_stream()" not in body:
                continue
            found += 1
            assert "__restrict__" not in signature + body and "__ldg" not in body, (name, signature)
    assert found == 4


def test_pairwise_fold_says_why_it_refuses_a_pointer(cuda_lib, capfd):
    assert cuda_lib.dccl_local_reduce_device(0x10002, 0x20000, 8, FLOAT32, OPS["sum"], None) != 0
    assert "between two elements of 4 bytes" in capfd.readouterr().err


def test_one_device_header_keeps_its_names(tmp_path):
    """As C, with every name that a caller may have sized something by."""
    src = tmp_path / "names.c"
    src.write_text("""#include "noalloc_allreduce.h"
unsigned sizes[] = {DCCL_NOALLOC_MAX_RANKS, DCCL_NOALLOC_MAX_BYTES, DCCL_NOALLOC_RANK_BYTES, DCCL_NOALLOC_SCRATCH_BYTES};
int codes[] = {DCCL_NOALLOC_OK, DCCL_NOALLOC_BAD_ARGUMENT, DCCL_NOALLOC_TOO_LARGE, DCCL_NOALLOC_CUDA_ERROR};
""")
    subprocess.run(["gcc", "-Wall", "-Werror", "-c", "-I", os.path.join(ROOT, "csrc", "kernels"), "-o", str(tmp_path / "names.o"), str(src)], check=True)
