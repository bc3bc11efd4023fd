"""Work that one GPU does for a user of this library, as cases that can be timed and checked.

Four families, each through the call a program makes:

``one_device``  ``dccl_allreduce_one_device_noalloc``: all-reduce among up to eight buffers of one device (model replicas or
                pipeline partitions driven by one process), from a handful of values to the entry point's limit of 256 KB.
``fold``        ``dccl_local_reduce_device``: acc = op(acc, in) on device buffers, the pairwise reduce a caller uses to
                accumulate gradients or partial results, from 256 KB to the 1 GiB messages of the benchmarks.
``copy``        a ``Communicator`` collective out of place in a world of one rank, which is what the same program runs on
                one GPU: all-reduce, reduce-scatter, all-gather, broadcast, all-to-all.
``zero``        ``ShardedOptimizer.step`` with AdamW: the update of 16-bit or 32-bit parameters from their fp32 masters.
"""
import ctypes
import math

import torch

from dccl_b200 import Communicator
from dccl_b200._lib import lib
from dccl_b200.comm import OPS, dtype_of
from dccl_b200.models.llama import Block, LlamaConfig, LlamaDecoder
from dccl_b200.parallel.zero import ShardedOptimizer

ONE_DEVICE_LIMIT = 256 << 10      # bytes per buffer that the entry point takes
BUCKET = 25 << 20                 # bytes of a gradient bucket, the default of GradientAllReducer
LARGEST = 1 << 30                 # bytes of the headline message
ADAMW = {"lr": 3e-4, "betas": (0.9, 0.95), "eps": 1e-8, "weight_decay": 0.1}


def listed():
    return [
        # eight replicas agree on a few scalars or a small norm vector: latency is everything
        {"name": "one_device_tiny", "kind": "one_device", "ranks": 8, "count": 256, "dtype": "float32", "op": "sum"},
        # three partitions average an activation of odd length
        {"name": "one_device_ragged", "kind": "one_device", "ranks": 3, "count": 10007, "dtype": "bfloat16", "op": "avg"},
        # eight replicas sum the largest buffers the entry point takes
        {"name": "one_device_limit", "kind": "one_device", "ranks": 8, "count": ONE_DEVICE_LIMIT // 4, "dtype": "float32", "op": "sum"},
        # the gradient of one small weight (2048 x 256 key projection) folded into its accumulator
        {"name": "fold_small", "kind": "fold", "count": 2048 * 256, "dtype": "bfloat16", "op": "sum"},
        # one gradient bucket accumulated in bf16
        {"name": "fold_bucket", "kind": "fold", "count": BUCKET // 2, "dtype": "bfloat16", "op": "sum"},
        # elementwise maximum over slices of flat fp16 buffers that start at odd elements
        {"name": "fold_view", "kind": "fold", "count": 6000011, "dtype": "float16", "op": "max", "acc_off": 1, "in_off": 3},
        # the largest message of the pairwise-reduce benchmark
        {"name": "fold_large", "kind": "fold", "count": LARGEST // 4, "dtype": "float32", "op": "sum"},
        # a loss value or a small norm on one GPU: launch cost
        {"name": "copy_small", "kind": "copy", "call": "all_reduce", "count": 1024, "dtype": "float32", "op": "sum"},
        # an all-gather out of a slice of a flat parameter buffer, ragged and not 16-byte aligned
        {"name": "copy_view", "kind": "copy", "call": "all_gather", "count": BUCKET // 2 + 13, "dtype": "bfloat16", "send_off": 3},
        # the headline message: 1 GiB of bf16
        {"name": "copy_large", "kind": "copy", "call": "all_reduce", "count": LARGEST // 2, "dtype": "bfloat16", "op": "sum"},
        # optimizer step of a model so small that launches dominate (the test configuration of the decoder, fp32)
        {"name": "zero_tiny", "kind": "zero", "model": "tiny", "dtype": "float32"},
        # optimizer step of one bf16 block of the training benchmark's decoder, 44 M parameters
        {"name": "zero_block", "kind": "zero", "model": "block", "dtype": "bfloat16"},
    ]


def _spread(rng, lo, hi):
    """A size between lo and hi, even over its logarithm, mostly odd."""
    v = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return max(lo, min(hi, v + (rng.random() < 0.5)))


def draw(rng):
    kind = rng.choice(["one_device", "one_device", "fold", "fold", "fold", "copy", "copy", "copy", "zero"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float32", "float32", "float16", "float64", "int32", "int64", "uint8", "int8"])
    size = torch.empty((), dtype=getattr(torch, dtype)).element_size()
    if kind == "one_device":
        return {"kind": kind, "ranks": rng.randint(2, 8), "count": _spread(rng, 5, ONE_DEVICE_LIMIT // size), "dtype": dtype,
                "op": rng.choice(["sum", "sum", "avg", "max", "min", "prod"]), "off": rng.choice([0, 0, 0, 1])}
    # slices at odd offsets are cut out of buckets; whole buffers go up to the largest message
    view = rng.random() < 0.4
    least = (256 << 10) if kind == "fold" else 4096
    count = _spread(rng, least // size, (BUCKET if view else LARGEST // 2) // size)
    if kind == "fold":
        return {"kind": kind, "count": count, "dtype": dtype, "op": rng.choice(["sum", "sum", "max", "min"]),
                "acc_off": rng.randint(0, 7) if view else 0, "in_off": rng.randint(0, 7) if view else 0}
    if kind == "copy":
        return {"kind": kind, "call": rng.choice(["all_reduce", "reduce_scatter", "all_gather", "broadcast", "all_to_all"]),
                "count": count, "dtype": dtype, "op": "sum", "send_off": rng.randint(0, 7) if view else 0}
    return {"kind": "zero", "model": "flat", "dtype": rng.choice(["bfloat16", "bfloat16", "float16", "float32"]),
            "rows": _spread(rng, 64, 8192), "cols": _spread(rng, 64, 4096)}


# -- inputs -----------------------------------------------------------------------------------------------------------

_comm = None


def _communicator():
    """The program's communicator: one rank, this GPU."""
    global _comm
    if _comm is None:
        _comm = Communicator(rank=0, world=1, device=torch.cuda.current_device())
    return _comm


def _values(count, dtype, gen):
    if dtype.is_floating_point:
        wide = dtype if dtype == torch.float64 else torch.float32
        out = torch.empty(count, dtype=dtype, device="cuda")
        # in pieces: the largest buffers are not held twice
        for lo in range(0, count, 1 << 26):
            n = min(count - lo, 1 << 26)
            out[lo:lo + n].copy_(torch.randn(n, dtype=wide, device="cuda", generator=gen))
        return out
    span = 12 if dtype in (torch.int8, torch.uint8) else 1000
    lo = 0 if dtype == torch.uint8 else -span
    return torch.randint(lo, span + 1, (count,), dtype=dtype, device="cuda", generator=gen)


def _buffer(count, dtype, gen, off=0):
    """`count` values that start `off` elements into an allocation."""
    return _values(count + off, dtype, gen)[off:]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _parameters(case, seed):
    """The parameters of a zero case, and two sets of gradients: one for the step before, one for the timed step."""
    dtype = getattr(torch, case["dtype"])
    torch.manual_seed(seed)
    with torch.device("cuda"):
        if case["model"] == "tiny":
            params = list(LlamaDecoder(LlamaConfig.tiny()).parameters())
        elif case["model"] == "block":
            params = list(Block(LlamaConfig.tinyllama_1b()).parameters())
        else:
            params = [torch.nn.Parameter(0.02 * torch.randn(case["rows"], case["cols"])), torch.nn.Parameter(torch.ones(case["cols"]))]
    for p in params:
        p.data = p.data.to(dtype)
    gen = _generator(seed)
    grads = [[(1e-3 * _values(p.numel(), torch.float32, gen)).to(dtype).view_as(p) for p in params] for _ in range(2)]
    return params, grads


def _operands(case, seed):
    dtype, gen = getattr(torch, case["dtype"]), _generator(seed)
    if case["kind"] == "one_device":
        return [_buffer(case["count"], dtype, gen, case.get("off", 0)) for _ in range(case["ranks"])]
    if case["kind"] == "fold":
        return [_buffer(case["count"], dtype, gen, case.get("acc_off", 0)), _buffer(case["count"], dtype, gen, case.get("in_off", 0))]
    return [_buffer(case["count"], dtype, gen, case.get("send_off", 0))]


def prepare(case, seed):
    s = {"kind": case["kind"], "stream": torch.cuda.current_stream().cuda_stream}
    if case["kind"] == "zero":
        params, grads = _parameters(case, seed)
        opt = ShardedOptimizer(params, _communicator(), **ADAMW)
        for g in grads:                         # a step before the timed one: its state exists and is not zero
            with torch.no_grad():
                for p, v in zip(params, g):
                    p.grad.copy_(v)
            if g is grads[0]:
                opt.step()
        return dict(s, opt=opt)
    ins = _operands(case, seed)
    s.update(ins=ins, dtype=dtype_of(ins[0]), count=case["count"])
    if case["kind"] == "one_device":
        fn = lib().dccl_allreduce_one_device_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_size_t, ctypes.POINTER(ctypes.c_void_p),
                       ctypes.POINTER(ctypes.c_void_p), ctypes.c_void_p, ctypes.c_void_p]
        outs = [torch.empty_like(x) for x in ins]
        table = ctypes.c_void_p * len(ins)
        s.update(fn=fn, op=OPS[case["op"]], outs=outs, in_table=table(*[x.data_ptr() for x in ins]), out_table=table(*[x.data_ptr() for x in outs]),
                 status=torch.empty(1, dtype=torch.int32, device="cuda"))
    elif case["kind"] == "fold":
        s.update(fn=lib().dccl_local_reduce_device, op=OPS[case["op"]])
    else:
        call = getattr(_communicator(), case["call"])
        kw = {"op": case["op"]} if case["call"] in ("all_reduce", "reduce_scatter") else {}
        s.update(call=call, kw=kw, out=torch.empty_like(ins[0]))
    return s


# -- one pass ---------------------------------------------------------------------------------------------------------

def run(s):
    if s["kind"] == "one_device":
        rc = s["fn"](len(s["ins"]), s["dtype"], s["op"], s["count"], s["in_table"], s["out_table"], s["status"].data_ptr(), s["stream"])
        if rc != 0:
            raise RuntimeError("one-device all-reduce returned %d" % rc)
        return {"out": s["outs"], "status": s["status"]}
    if s["kind"] == "fold":
        acc, x = s["ins"]
        if s["fn"](acc.data_ptr(), x.data_ptr(), s["count"], s["dtype"], s["op"], s["stream"]) != 0:
            raise RuntimeError("pairwise reduce failed")
        return {"acc": acc}
    if s["kind"] == "copy":
        return {"out": s["call"](s["ins"][0], s["out"], **s["kw"])}
    opt = s["opt"]
    opt.step()
    out = []
    for g in opt.groups:
        st = opt.inner.state[g["master"]]
        out.append({"params": g["flat"], "master": g["master"].detach(), "exp_avg": st["exp_avg"], "exp_avg_sq": st["exp_avg_sq"]})
    return out


def work(case):
    size = torch.empty((), dtype=getattr(torch, case["dtype"])).element_size()
    if case["kind"] == "zero":
        n = _parameter_count(case)
        # gradient in, parameter out, and master, first and second moment in fp32 both ways
        return {"bytes": n * (2 * size + 24), "flops": 14 * n}
    nbytes = case["count"] * size
    if case["kind"] == "one_device":
        return {"bytes": 2 * case["ranks"] * nbytes, "flops": (case["ranks"] - 1) * case["count"]}
    if case["kind"] == "fold":
        return {"bytes": 3 * nbytes, "flops": case["count"]}
    return {"bytes": 2 * nbytes, "flops": 0}


def _parameter_count(case):
    if case["model"] == "flat":
        return case["rows"] * case["cols"] + case["cols"]
    cfg = LlamaConfig.tiny() if case["model"] == "tiny" else LlamaConfig.tinyllama_1b()
    whole = cfg.num_params()
    if case["model"] == "tiny":
        return whole
    return (whole - 2 * cfg.vocab_size * cfg.hidden - cfg.hidden) // cfg.layers


def tolerance(case):
    if case["kind"] == "copy" or not getattr(torch, case["dtype"]).is_floating_point or case.get("op") in ("max", "min"):
        return "exact"
    # One rounding to the result's type, after sums of up to eight values (or an update) in that type or in fp32.
    # rel: four times the relative error measured against 64 bits; max: one unit in the last place of the result's type
    # (16-bit types), or a few roundings of the sums.
    return {"float64": {"rel": 1e-15, "max": 1e-14}, "float32": {"rel": 2.5e-7, "max": 2e-6},
            "float16": {"rel": 1e-3, "max": 2e-3}, "bfloat16": {"rel": 7e-3, "max": 8e-3}}[case["dtype"]]


# -- the same in 64 bits ----------------------------------------------------------------------------------------------

def exact(case, seed):
    if case["kind"] == "zero":
        return _exact_adamw(case, seed)
    ins = _operands(case, seed)
    if not ins[0].dtype.is_floating_point:
        return None
    if case["kind"] == "copy":
        return {"out": ins[0]}
    acc = ins[0].double()
    for x in ins[1:]:
        x = x.double()
        acc = {"sum": torch.add, "avg": torch.add, "prod": torch.mul, "max": torch.maximum, "min": torch.minimum}[case["op"]](acc, x)
    if case["kind"] == "fold":
        return {"acc": acc}
    if case["op"] == "avg":
        acc = acc / len(ins)
    return {"out": [acc] * len(ins), "status": None}


def _exact_adamw(case, seed):
    params, grads = _parameters(case, seed)
    align = 16 // params[0].element_size()
    flat = lambda ts: torch.cat([torch.nn.functional.pad(t.detach().reshape(-1).double(), (0, -t.numel() % align)) for t in ts])  # noqa: E731
    p = flat(params)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    b1, b2 = ADAMW["betas"]
    for t, gs in enumerate(grads, 1):
        g = flat(gs)
        p = p * (1 - ADAMW["lr"] * ADAMW["weight_decay"])
        m = b1 * m + (1 - b1) * g
        v = b2 * v + (1 - b2) * g * g
        p = p - ADAMW["lr"] / (1 - b1 ** t) * m / ((v / (1 - b2 ** t)).sqrt() + ADAMW["eps"])
    return [{"params": p, "master": p, "exp_avg": m, "exp_avg_sq": v}]
