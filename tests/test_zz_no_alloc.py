"""The entry point that allocates nothing (csrc/kernels/noalloc_allreduce.h).

Some callers of the library may not allocate device memory when they need a reduction: all of it
may be handed out to a caching allocator or a KV-cache pool, or they sit on a path where the
device-wide synchronisation of cudaMalloc is not acceptable. For them the library exports
dccl_allreduce_one_device_noalloc, an all-reduce among buffers on one device that needs no scratch.
This test calls it through its exported C symbol, the way
such a caller would, twice in a row on the same stream, and compares every rank's output with
what the allocating entry point (dccl_emu_collective, two-shot variant) returns for the same
inputs, and with a fold of the inputs computed on the CPU in fp64 / int64 (the two kernels share
their reduction code, so agreement between them alone would not show a fault in it). The buffers the TEST needs are made with torch; the entry point under test gets only
their addresses. The file sorts last so that a run that stops at the first failure has already
run everything else; it also passes when run alone in a fresh process.
"""
import ctypes

import numpy as np
import pytest

from dccl_b200.comm import DTYPE_NAMES, OPS
from dccl_b200.utils import oracle

pytestmark = pytest.mark.gpu

MAX_BYTES = 256 * 1024


def _entry(lib):
    fn = lib.dccl_allreduce_one_device_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_size_t, ctypes.POINTER(ctypes.c_void_p),
                   ctypes.POINTER(ctypes.c_void_p), ctypes.c_void_p, ctypes.c_void_p]
    return fn


def _reference(lib, n, name, op, count, ins):
    """Outputs of the existing (allocating) entry point: [n, count]."""
    np_dt = np.dtype(np.uint16) if name == "bfloat16" else np.dtype(name)
    hin = np.concatenate(ins).astype(np_dt, copy=False)
    hout = np.zeros(n * count, dtype=np_dt)
    rc = lib.dccl_emu_collective(b"allreduce", b"twoshot", n, DTYPE_NAMES.index(name), OPS[op], count, 0, 4, 0, 0, 1, 0,
                                 hin.ctypes.data, hout.ctypes.data)
    assert rc == 0
    return hout.reshape(n, count)


def _close(got, want, name, n):
    rtol, atol = oracle.tolerances(name, n)
    if rtol == 0.0:
        return np.array_equal(got, want)
    if name == "bfloat16":
        got, want = oracle.bf16_to_f32(got), oracle.bf16_to_f32(want)
    return np.allclose(got.astype(np.float64), want.astype(np.float64), rtol=rtol, atol=atol)


def _run(lib, torch, n, name, op, count, seed, in_place=False):
    fn = _entry(lib)
    np_dt = np.dtype(np.uint16) if name == "bfloat16" else np.dtype(name)
    ins = [oracle.make_input(name, count, seed=seed * 10 + r) for r in range(n)]
    want = _reference(lib, n, name, op, count, ins)
    # device buffers for the call under test (bit patterns travel as integers of the same width)
    carrier = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[np_dt.itemsize]
    d_in = [torch.from_numpy(x.view({1: np.uint8, 2: np.int16, 4: np.int32, 8: np.int64}[np_dt.itemsize]).copy()).to("cuda") for x in ins]
    d_out = d_in if in_place else [torch.full((count,), 0x55, dtype=carrier, device="cuda") for _ in range(n)]
    status = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    in_ptrs = (ctypes.c_void_p * n)(*[t.data_ptr() for t in d_in])
    out_ptrs = (ctypes.c_void_p * n)(*[t.data_ptr() for t in d_out])
    stream = torch.cuda.current_stream().cuda_stream
    rc = fn(n, DTYPE_NAMES.index(name), OPS[op], count, in_ptrs, out_ptrs, status.data_ptr(), stream)
    assert rc == 0, "entry point returned %d" % rc
    torch.cuda.synchronize()
    assert int(status.item()) == 0, "a wait inside the kernel gave up"
    serial = oracle.fold(ins, op, bf16=name == "bfloat16")      # independent of any kernel of the library
    for r in range(n):
        got = d_out[r].cpu().numpy().view(np_dt)
        assert _close(got, want[r], name, n), (n, name, op, count, r)
        assert _close(got, serial, name, n), ("against the serial fold", n, name, op, count, r)


def test_two_calls_in_a_row_match_the_allocating_entry_point(dccl_lib):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    torch.cuda.set_device(0)
    # two calls of different shapes, so that anything left over from the first would show
    _run(dccl_lib, torch, 8, "float32", "sum", MAX_BYTES // 4, seed=1)
    _run(dccl_lib, torch, 3, "bfloat16", "avg", 10007, seed=2)
    # and more pairs: every width, in place, one rank, tiny messages
    _run(dccl_lib, torch, 4, "int32", "max", 4099, seed=3)
    _run(dccl_lib, torch, 4, "int32", "max", 4099, seed=4, in_place=True)
    _run(dccl_lib, torch, 2, "float64", "prod", 1000, seed=5)
    _run(dccl_lib, torch, 1, "float16", "sum", 5, seed=6)
    _run(dccl_lib, torch, 5, "uint8", "min", 3, seed=7)
    _run(dccl_lib, torch, 2, "float32", "sum", MAX_BYTES // 4, seed=8)   # the limit with the fewest ranks


def test_requests_beyond_the_limits_are_refused(dccl_lib, capfd):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    fn = _entry(dccl_lib)
    t = torch.zeros(16, dtype=torch.float32, device="cuda")
    ptrs = (ctypes.c_void_p * 2)(t.data_ptr(), t.data_ptr())
    assert fn(2, 7, 0, MAX_BYTES // 4 + 1, ptrs, ptrs, None, None) == -2     # too large: nothing is launched
    assert "above the limit" in capfd.readouterr().err
    assert fn(9, 7, 0, 4, ptrs, ptrs, None, None) == -1                        # more ranks than the limit
    assert fn(2, 7, 0, 0, ptrs, ptrs, None, None) == 0                         # nothing to do
    torch.cuda.synchronize()


@pytest.mark.parametrize("n,name,op,count,off", [
    (8, "float32", "sum", 1, 0),                       # one element: no vector at all
    (3, "float32", "sum", 4 * 128 + 3, 0),             # one full CTA of vectors and a tail
    (5, "bfloat16", "sum", 1003, 1),                   # head of 7, vectors that cross shard ends
    (7, "float16", "avg", 40, 3),                      # shards of one vector
    (4, "int8", "prod", 4097, 5),
    (2, "float64", "sum", MAX_BYTES // 8, 1),          # the limit behind a head of one element
    (8, "uint8", "max", MAX_BYTES, 0),
])
@pytest.mark.parametrize("form", ["apart", "in_place", "crossed", "uneven"])
def test_one_pass_equals_the_two_shot_fold_bit_for_bit(dccl_lib, n, name, op, count, off, form):
    """Heads, tails, shard ends inside a vector, outputs that are another rank's input, and buffers whose distances to a
    16-byte boundary differ. The fold order is the two-shot kernel's, so results are compared as bits."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    np_dt = np.dtype(np.uint16) if name == "bfloat16" else np.dtype(name)
    ins = [oracle.make_input(name, count, seed=50 + r) for r in range(n)]
    want = _reference(dccl_lib, n, name, op, count, ins)
    np_carrier = {1: np.uint8, 2: np.int16, 4: np.int32, 8: np.int64}[np_dt.itemsize]
    carrier = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[np_dt.itemsize]
    offs = [off + (r % 2 if form == "uneven" else 0) for r in range(n)]
    d_in = []
    for x, o in zip(ins, offs):
        buf = torch.zeros(count + o, dtype=carrier, device="cuda")
        buf[o:].copy_(torch.from_numpy(x.view(np_carrier).copy()))
        d_in.append(buf[o:])
    guard = [torch.full((count + off + 8,), 0x55, dtype=carrier, device="cuda") for _ in range(n)]
    d_out = d_in if form == "in_place" else d_in[1:] + d_in[:1] if form == "crossed" else [g[off:off + count] for g in guard]
    status = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    rc = _entry(dccl_lib)(n, DTYPE_NAMES.index(name), OPS[op], count, (ctypes.c_void_p * n)(*[t.data_ptr() for t in d_in]),
                          (ctypes.c_void_p * n)(*[t.data_ptr() for t in d_out]), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for r in range(n):
        assert np.array_equal(d_out[r].cpu().numpy().view(np_dt).view(np_carrier), want[r].view(np_carrier)), r
    for g in guard:      # nothing before or behind the outputs
        assert torch.all(g[:off] == 0x55) and torch.all(g[off + count:] == 0x55)


@pytest.mark.parametrize("name", ["int8", "uint8"])
@pytest.mark.parametrize("op", ["sum", "avg", "max", "min", "prod"])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 8])
def test_bytes_of_the_whole_range(dccl_lib, name, op, n):
    """Whole vectors of bytes fold four at a time and divide by multiplying: every value, wrapping sums, both signs."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    rng = np.random.default_rng(n)
    count = 2048 + 5
    ins = [rng.integers(0, 256, count).astype(np.uint8).view(name) for _ in range(n)]
    ins[0][:256] = np.arange(256).astype(np.uint8).view(name)
    for x in ins[1:]:
        x[:256] = 0                                  # every value once, divided by n
    want = oracle.fold(ins, op)
    d_in = [torch.from_numpy(x.view(np.uint8).copy()).to("cuda") for x in ins]
    d_out = [torch.empty_like(x) for x in d_in]
    rc = _entry(dccl_lib)(n, DTYPE_NAMES.index(name), OPS[op], count, (ctypes.c_void_p * n)(*[t.data_ptr() for t in d_in]),
                          (ctypes.c_void_p * n)(*[t.data_ptr() for t in d_out]), None, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    for t in d_out:
        assert np.array_equal(t.cpu().numpy().view(name), want)
    if n == 2:                                        # the pairwise fold of the same bytes (an average accumulates like a sum)
        rc = dccl_lib.dccl_local_reduce_device(d_in[0].data_ptr(), d_in[1].data_ptr(), count, DTYPE_NAMES.index(name), OPS[op],
                                               torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and np.array_equal(d_in[0].cpu().numpy().view(name), oracle.fold(ins, "sum" if op == "avg" else op))


@pytest.mark.parametrize("name,count", [("float32", 1), ("bfloat16", 1003), ("float64", MAX_BYTES // 8)])
@pytest.mark.parametrize("in_off,out_off", [(1, 1), (0, 1), (3, 6), (5, 5)])
def test_one_rank_copies_from_and_to_any_address(dccl_lib, name, count, in_off, out_off):
    """Addresses between two elements included: a copy has no elements."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    nbytes = count * np.dtype("uint16" if name == "bfloat16" else name).itemsize
    src = torch.randint(0, 255, (nbytes + 16,), dtype=torch.uint8, device="cuda")
    dst = torch.full((nbytes + 16,), 0xAB, dtype=torch.uint8, device="cuda")
    want = dst.clone()
    want[out_off:out_off + nbytes] = src[in_off:in_off + nbytes]
    rc = _entry(dccl_lib)(1, DTYPE_NAMES.index(name), OPS["sum"], count, (ctypes.c_void_p * 1)(src.data_ptr() + in_off),
                          (ctypes.c_void_p * 1)(dst.data_ptr() + out_off), None, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(dst, want)


def _call(lib, torch, ins, outs, stream):
    n = len(ins)
    rc = _entry(lib)(n, DTYPE_NAMES.index("float32"), OPS["sum"], ins[0].numel(), (ctypes.c_void_p * n)(*[t.data_ptr() for t in ins]),
                     (ctypes.c_void_p * n)(*[t.data_ptr() for t in outs]), None, stream.cuda_stream)
    assert rc == 0


def test_calls_on_different_streams_overlap(dccl_lib):
    """Three streams, each with chains of its own calls and nothing that orders them: calls share no state."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    streams = [torch.cuda.Stream() for _ in range(3)]
    # whole numbers, which are exact: in place, every call after a chain's first multiplies by the number of ranks
    bufs = [[torch.full((MAX_BYTES // 4 - s,), float(10 * s + r), device="cuda") for r in range(4)] for s in range(3)]
    torch.cuda.synchronize()
    for s in streams:
        with torch.cuda.stream(s):
            torch.cuda._sleep(1000000)              # all chains are queued before the first runs
    for k in range(4):
        for s, b in zip(streams, bufs):
            _call(dccl_lib, torch, b, b, s)
    torch.cuda.synchronize()
    for s, b in enumerate(bufs):
        for t in b:
            assert torch.all(t == 64.0 * (40 * s + 6))


def test_calls_are_captured_in_a_graph(dccl_lib):
    """Two that depend on each other, replayed on new values."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    ins = [torch.zeros(10007, device="cuda") for _ in range(5)]
    outs = [torch.empty_like(t) for t in ins]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _call(dccl_lib, torch, ins, outs, torch.cuda.current_stream())
        _call(dccl_lib, torch, outs, ins, torch.cuda.current_stream())
    for k in range(1, 4):
        for r, t in enumerate(ins):
            t.fill_(float(k * r))
        graph.replay()
        for o, i in zip(outs, ins):
            assert torch.all(o == 10.0 * k) and torch.all(i == 50.0 * k)
