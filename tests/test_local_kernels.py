"""The one-rank copy and the pairwise fold on device buffers at every distance from a 16-byte boundary, at lengths around
the vector and CTA sizes: results are exact, and nothing around the destination is touched."""
import os

import pytest

torch = pytest.importorskip("torch")

from dccl_b200 import Communicator  # noqa: E402
from dccl_b200.comm import OPS, dtype_of  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm(dccl_lib):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    saved = dict(os.environ)
    c = Communicator(rank=0, world=1, device=0)
    yield c
    c.finalize()
    os.environ.clear()
    os.environ.update(saved)


@pytest.mark.parametrize("nbytes", [1, 15, 16, 17, 31, 48, 63, 79, 200, 8191, 8192, 8193, 8192 + 63, 3 * 8192 + 31, 1 << 20])
def test_copy_at_every_pair_of_offsets(comm, nbytes):
    gen = torch.Generator(device="cuda").manual_seed(nbytes)
    src = torch.randint(0, 255, (nbytes + 32,), dtype=torch.uint8, device="cuda", generator=gen)
    offsets = (0, 1, 3, 4, 6, 8, 13, 15)
    for so in offsets:
        for do in offsets:
            dst = torch.full((nbytes + 32,), 0xAB, dtype=torch.uint8, device="cuda")
            comm.all_gather(src[so:so + nbytes], dst[do:do + nbytes])
            want = torch.full_like(dst, 0xAB)
            want[do:do + nbytes] = src[so:so + nbytes]
            assert torch.equal(dst, want), (nbytes, so, do)


@pytest.mark.parametrize("nbytes", [(80 << 20) - 1, 80 << 20, (80 << 20) + 32768 + 17])
def test_copy_where_its_ctas_grow(comm, nbytes):
    test_copy_where_its_shape_changes(comm, nbytes)


@pytest.mark.parametrize("nbytes", [(28 << 20) - 1, 28 << 20, (28 << 20) + 32768 + 17])
def test_copy_where_its_shape_changes(comm, nbytes):
    src = torch.randint(0, 255, (nbytes + 32,), dtype=torch.uint8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(nbytes))
    for so, do in ((0, 0), (6, 0), (0, 1), (3, 13)):
        dst = torch.full((nbytes + 32,), 0xAB, dtype=torch.uint8, device="cuda")
        comm.all_gather(src[so:so + nbytes], dst[do:do + nbytes])
        assert torch.equal(dst[do:do + nbytes], src[so:so + nbytes])
        assert bool((dst[:do] == 0xAB).all()) and bool((dst[do + nbytes:] == 0xAB).all())


@pytest.mark.parametrize("dtype", [torch.int8, torch.uint8, torch.int32, torch.int64, torch.float16, torch.bfloat16, torch.float32, torch.float64])
@pytest.mark.parametrize("op", ["sum", "prod", "max", "min"])
def test_fold_at_every_pair_of_offsets(dccl_lib, dtype, op):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    ve = 16 // torch.empty((), dtype=dtype).element_size()
    stream = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(5)
    for count in (1, 3 * ve + 1, 512 * ve, 512 * ve + ve + 3):
        x = torch.randint(0, 12, (count + ve,), device="cuda", generator=gen).to(dtype)
        a = torch.randint(0, 12, (count + ve,), device="cuda", generator=gen).to(dtype)      # products stay in the 8-bit range
        if dtype.is_floating_point:
            x += torch.rand(count + ve, device="cuda", generator=gen).to(dtype)
            x[0], x[count // 2], a[count // 3] = float("inf"), float("nan"), float("-inf")
        for ao in sorted({0, 1, ve // 2, ve - 1}):
            for xo in sorted({0, 1, ve // 2, ve - 1}):
                acc = a.clone()
                rc = dccl_lib.dccl_local_reduce_device(acc[ao:].data_ptr(), x[xo:].data_ptr(), count, dtype_of(acc), OPS[op], stream)
                assert rc == 0
                p, q = a[ao:ao + count], x[xo:xo + count]
                # 16-bit types: fp32 and one rounding, which is what torch's own operators do; a NaN loses to a number in max / min
                if dtype.is_floating_point and op in ("max", "min"):
                    r = torch.fmax(p, q) if op == "max" else torch.fmin(p, q)
                else:
                    r = {"sum": torch.add, "prod": torch.mul, "max": torch.maximum, "min": torch.minimum}[op](p, q)
                want = a.clone()
                want[ao:ao + count] = r
                assert torch.equal(torch.nan_to_num(acc), torch.nan_to_num(want)) and torch.equal(acc.isnan(), want.isnan()), (count, ao, xo)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("op", ["sum", "max", "min"])
def test_pairs_of_16_bit_floats_fold_as_they_do_one_by_one(dccl_lib, dtype, op):
    """Every bit pattern against every 29th one and the special ones, in both orders."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    every = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype)
    some = [0, 1, 0x03FF, 0x0400, 0x7BFF, 0x7C00, 0x7C01, 0x7E00, 0x7F7F, 0x7F80, 0x7F81, 0x7FFF, 0x007F, 0x0080]
    some = torch.tensor(some + [s - 0x8000 for s in some] + list(range(-32768, 32768, 29)), device="cuda", dtype=torch.int32).to(torch.int16).view(dtype)
    stream = torch.cuda.current_stream().cuda_stream
    for part in some.split(256):
        x = every.repeat(part.numel())
        a = part.repeat_interleave(every.numel())
        for first, second in ((a, x), (x, a)):
            acc, p, q = first.clone(), first.float(), second.float()
            assert dccl_lib.dccl_local_reduce_device(acc.data_ptr(), second.data_ptr(), acc.numel(), dtype_of(acc), OPS[op], stream) == 0
            if op == "sum":
                want = (p + q).to(dtype)
            else:                                                # of equal values, two zeros among them, the first; a NaN loses to a number
                want = torch.where(((p < q) if op == "max" else (q < p)) | p.isnan(), second, first)
            nan = want.isnan()
            assert torch.equal(acc.isnan(), nan)
            assert torch.equal(acc.view(torch.int16).masked_fill(nan, 0), want.view(torch.int16).masked_fill(nan, 0))


@pytest.mark.parametrize("edge", [10 << 20, 22 << 20])
@pytest.mark.parametrize("dtype", [torch.int8, torch.bfloat16, torch.float32, torch.float64])
def test_fold_where_its_shape_changes(dccl_lib, dtype, edge):
    """Below, at and above the sizes between which a thread folds two vectors; ends of every kind; nothing else is touched."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    es = torch.empty((), dtype=dtype).element_size()
    stream = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(edge)
    room = edge // es + 8192
    x = torch.randint(-50, 50, (room,), device="cuda", generator=gen).to(dtype)      # sums of two are exact in every type
    a = torch.randint(-50, 50, (room,), device="cuda", generator=gen).to(dtype)
    for count in (edge // es - 1, edge // es, edge // es + 1, edge // es + 4096 // es + 3):
        for ao, xo in ((0, 0), (0, 3), (1, 0), (3, 1)):
            acc, want = a.clone(), a.clone()
            assert dccl_lib.dccl_local_reduce_device(acc[ao:].data_ptr(), x[xo:].data_ptr(), count, dtype_of(acc), OPS["sum"], stream) == 0
            want[ao:ao + count] += x[xo:xo + count]
            assert torch.equal(acc, want), (count, ao, xo)


def test_fold_into_itself_and_pointers_between_elements(dccl_lib):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    stream = torch.cuda.current_stream().cuda_stream
    a = torch.arange(5003, dtype=torch.float32, device="cuda")[3:]
    want = a + a
    assert dccl_lib.dccl_local_reduce_device(a.data_ptr(), a.data_ptr(), a.numel(), dtype_of(a), OPS["sum"], stream) == 0
    assert torch.equal(a, want)
    assert dccl_lib.dccl_local_reduce_device(a.data_ptr() + 2, a.data_ptr(), 8, dtype_of(a), OPS["sum"], stream) != 0
    assert torch.equal(a, want)


def test_copy_and_fold_are_captured_and_replayed(comm, dccl_lib):
    """Back to back on one stream, eager and from a graph: each call sees what the one before it wrote."""
    n = (1 << 20) + 5
    x = torch.arange(n, dtype=torch.float32, device="cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)

    def chain():
        stream = torch.cuda.current_stream().cuda_stream
        comm.all_reduce(x, a)                                                                                   # a = x
        assert dccl_lib.dccl_local_reduce_device(a.data_ptr(), x.data_ptr(), n, dtype_of(a), OPS["sum"], stream) == 0   # a = 2x
        comm.all_reduce(a, b)
        assert dccl_lib.dccl_local_reduce_device(b.data_ptr(), a.data_ptr(), n, dtype_of(a), OPS["sum"], stream) == 0   # b = 4x
        x.add_(1.0)

    for k in range(8):
        chain()
        assert torch.equal(b, 4 * (x - 1))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for k in range(8):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(b, 4 * (x - 1)) and float(x[0]) == 16.0


def test_calls_wait_for_other_streams_and_for_copies_and_fills(comm, dccl_lib):
    """An event of another stream, a copy or a fill between two calls is waited for like by any kernel."""
    n = 1 << 20
    x, y, a = (torch.zeros(n, device="cuda") for _ in range(3))
    host = torch.empty(n, pin_memory=True)
    side = torch.cuda.Stream()
    here = torch.cuda.current_stream()
    for k in range(1, 21):
        comm.all_reduce(x, a)                       # a call right before, so that the next one could be set up early
        side.wait_stream(here)
        with torch.cuda.stream(side):
            torch.cuda._sleep(200000)
            x.fill_(float(k))
        here.wait_stream(side)
        comm.all_reduce(x, y)                       # reads what the other stream has just written
        host.fill_(float(k))
        a.copy_(host, non_blocking=True)            # a copy, then a fold of its destination
        assert dccl_lib.dccl_local_reduce_device(a.data_ptr(), y.data_ptr(), n, dtype_of(a), OPS["sum"], here.cuda_stream) == 0
        assert torch.equal(a, torch.full_like(a, 2.0 * k)) and torch.equal(y, torch.full_like(y, float(k))), k
