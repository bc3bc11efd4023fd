"""Kernels that are launched while the kernel before them still runs read what that kernel has yet to write: behind a kernel
that lets the next launch start at once and writes 300 us later."""
import ctypes

import pytest

torch = pytest.importorskip("torch")

from dccl_b200 import Communicator  # noqa: E402
from dccl_b200.comm import OPS, dtype_of  # noqa: E402
from dccl_b200.parallel import zero  # noqa: E402

pytestmark = pytest.mark.gpu

WORDS = 1 << 18
SPIN_US = 300


@pytest.fixture
def late(dccl_lib):
    """late(dst, src): dst = src on the current stream, late."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")

    def call(dst, src, end=None):
        assert dst.nbytes == src.nbytes
        rc = dccl_lib.dccl_emu_early_producer(dst.data_ptr(), src.data_ptr(), dst.nbytes // 4, SPIN_US, end.data_ptr() if end is not None else None,
                                              torch.cuda.current_stream().cuda_stream)
        assert rc == 0

    return call


def test_the_next_launch_does_start_early(dccl_lib, late):
    """What the other tests rely on: the kernel behind the producer runs before the producer has written. (It may; one of
    several tries is enough.)"""
    src, dst = torch.ones(WORDS, device="cuda"), torch.zeros(WORDS, device="cuda")
    times = torch.zeros(2, 8, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for k in range(8):
        late(dst, src, times[0, k:])
        assert dccl_lib.dccl_emu_early_observer(times[1, k:].data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    end, start = times.cpu()
    assert (start < end).any(), (start - end).tolist()


@pytest.mark.parametrize("offset", [0, 3])      # whole vectors, and the window over two of them
def test_copy_and_fold_read_what_the_kernel_before_them_writes(dccl_lib, late, offset):
    comm = Communicator(rank=0, world=1, device=0)
    try:
        src = torch.randint(-1000, 1000, (WORDS,), dtype=torch.int32, device="cuda")
        buf, out = torch.zeros_like(src), torch.empty_like(src)
        n = WORDS - offset
        torch.cuda.synchronize()
        for k in range(5):
            late(buf, src)
            comm.all_reduce(buf[offset:], out[:n])
            assert torch.equal(out[:n], src[offset:])
            acc = torch.zeros_like(src)
            buf.zero_()
            late(buf, src)
            stream = torch.cuda.current_stream().cuda_stream
            assert dccl_lib.dccl_local_reduce_device(acc.data_ptr(), buf[offset:].data_ptr(), n, dtype_of(acc), OPS["sum"], stream) == 0
            assert torch.equal(acc[:n], src[offset:])
            late(acc, src)                      # the accumulator, too
            assert dccl_lib.dccl_local_reduce_device(acc.data_ptr(), src.data_ptr(), n, dtype_of(acc), OPS["sum"], stream) == 0
            assert torch.equal(acc[:n], 2 * src[:n])
            buf.zero_()
            src += 1
    finally:
        comm.finalize()


@pytest.mark.parametrize("offsets", [(0, 0, 0), (0, 1, 2)])      # vectors, and elements one by one
def test_one_device_all_reduce_reads_what_the_kernel_before_it_writes(dccl_lib, late, offsets):
    fn = dccl_lib.dccl_allreduce_one_device_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    count, n = 8192, len(offsets)
    src = torch.randint(-1000, 1000, (n, count + 4), dtype=torch.int32, device="cuda")
    buf, out = torch.zeros_like(src), torch.empty_like(src)
    ins = (ctypes.c_void_p * n)(*[buf[r, o:].data_ptr() for r, o in enumerate(offsets)])
    outs = (ctypes.c_void_p * n)(*[out[r].data_ptr() for r in range(n)])
    torch.cuda.synchronize()
    for k in range(5):
        late(buf, src)
        assert fn(n, dtype_of(src), OPS["sum"], count, ins, outs, None, torch.cuda.current_stream().cuda_stream) == 0
        want = sum(src[r, o:o + count] for r, o in enumerate(offsets))
        assert torch.equal(out[:, :count], want.expand(n, count))
        buf.zero_()
        src += 1


@pytest.mark.parametrize("offset", [0, 1])      # whole vectors, and state that is not aligned
def test_adamw_reads_what_the_kernel_before_it_writes(dccl_lib, late, offset):
    n = 4096
    old, new = torch.ones(n + offset, device="cuda"), torch.full((n + offset,), 2.0, device="cuda")
    grad = torch.zeros(n, device="cuda")
    p, master_grad, out = (torch.zeros(n, device="cuda") for _ in range(3))
    m, v = torch.zeros(n + offset, device="cuda"), torch.zeros(n + offset, device="cuda")
    torch.cuda.synchronize()
    for k in range(5):
        for t in (p, m, v):
            t.copy_(old[:t.numel()])
        grad.zero_()
        late(m, new)                            # not the last one before the update: done when that one is
        late(grad, new[:n])
        rc = dccl_lib.dccl_adamw_flat(0, dtype_of(grad), n, p.data_ptr(), master_grad.data_ptr(), m[offset:].data_ptr(), v[offset:].data_ptr(), grad.data_ptr(),
                                      out.data_ptr(), 1.0, 0.5, 0.5, 0.5, 1.0, 1.0, 0.0, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        # m = 2 + (2 - 2) / 2, v = 1 / 2 + 4 / 2, p = 1 - m / sqrt(v)
        assert torch.equal(master_grad, grad) and float(grad[0]) == 2.0
        torch.testing.assert_close(out, torch.full_like(out, 1 - 2 / 2.5 ** 0.5), rtol=0, atol=2.0 ** -21)
        assert torch.equal(out, p)


def test_calls_on_the_legacy_stream_wait_for_blocking_streams(dccl_lib, late):
    """The legacy default stream waits for work on streams that were created as blocking ones, without any event."""
    comm = Communicator(rank=0, world=1, device=0)
    handle = ctypes.c_ulonglong(0)
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
    try:
        blocking = torch.cuda.ExternalStream(handle.value)
        x, y = torch.zeros(WORDS, device="cuda"), torch.zeros(WORDS, device="cuda")
        assert torch.cuda.current_stream().cuda_stream == 0
        torch.cuda.synchronize()
        for k in range(1, 11):
            comm.all_reduce(x, y)               # a call right before, so that the next one could be set up early
            with torch.cuda.stream(blocking):
                torch.cuda._sleep(200000)
                x.fill_(float(k))
            comm.all_reduce(x, y)
            assert torch.all(y == float(k))
    finally:
        torch.cuda.synchronize()
        torch.cuda.cudart().cudaStreamDestroy(handle.value)
        comm.finalize()
