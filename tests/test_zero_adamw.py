"""The one-kernel AdamW update of dccl_b200.parallel.zero against the general path (torch's own optimizer and the casts
around it), and which optimizers may take it."""
import collections
import ctypes
import functools
import os
import re
import warnings

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from torch.optim.optimizer import register_optimizer_step_post_hook, register_optimizer_step_pre_hook  # noqa: E402
from torch.overrides import TorchFunctionMode  # noqa: E402
from torch.utils._python_dispatch import TorchDispatchMode  # noqa: E402

from dccl_b200.parallel import zero  # noqa: E402


class OneProcess:
    """The collectives of a world whose other ranks hold the same gradients (world 1 or 2), on the current device."""

    rank, has_multicast = 0, False

    def __init__(self, world):
        self.world = world

    def reduce_scatter(self, send, recv, op="sum"):
        recv.copy_(send[:recv.numel()])

    def all_gather(self, send, recv):
        recv[:send.numel()].copy_(send)


def _make(world, dtype, sizes, general, device="cuda", cls=torch.optim.AdamW, **kw):
    torch.manual_seed(3)
    params = [torch.nn.Parameter(torch.randn(s).to(dtype).to(device)) for s in sizes]
    opt = zero.ShardedOptimizer(params, OneProcess(world), cls, symmetric=False, **dict(dict(lr=1e-2, betas=(0.9, 0.95), weight_decay=0.1), **kw))
    if general:
        opt.inner.register_step_pre_hook(lambda *a: None)      # anything hooked into the step keeps the general path
    return opt


def _train(opt, steps, scheduler=False):
    sched = torch.optim.lr_scheduler.LambdaLR(opt.inner, lambda t: 0.5 ** t) if scheduler else None
    for s in range(steps):
        for i, g in enumerate(opt.groups):
            gen = torch.Generator().manual_seed(100 * s + i)
            g["grad"].copy_(torch.randn(g["grad"].numel(), generator=gen) * 10.0 ** (s - 2))
        opt.step()
        if sched:
            sched.step()
    return opt


@pytest.mark.gpu
@pytest.mark.parametrize("world", [1, 2])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sizes", [[3], [2048, 1], [2049 * 5, 7]])           # below one vector, one CTA, several and a tail
@pytest.mark.parametrize("kw", [{}, {"betas": (0.0, 0.5), "weight_decay": 0.0}, {"betas": (0.4, 0.999), "scheduler": True}])
def test_one_kernel_update_matches_the_general_path(dccl_lib, world, dtype, sizes, kw):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    kw, steps = dict(kw), 4
    scheduler = kw.pop("scheduler", False)
    a, b = (_train(_make(world, dtype, sizes, general, **kw), steps, scheduler) for general in (False, True))
    assert a._adamw_updates() is not None and b._adamw_updates() is None
    ga, gb = a.groups[0], b.groups[0]
    sa, sb = a.inner.state[ga["master"]], b.inner.state[gb["master"]]
    u = 2.0 ** -23
    assert float(sa["step"]) == float(sb["step"]) == steps
    assert torch.equal(ga["master"].grad, gb["master"].grad)
    # every step rounds each moment a few times, relative to the gradients it mixes (up to 10 x 4 sigma, and their squares)
    torch.testing.assert_close(sa["exp_avg"], sb["exp_avg"], rtol=4 * steps * u, atol=4 * steps * u * 50)
    torch.testing.assert_close(sa["exp_avg_sq"], sb["exp_avg_sq"], rtol=4 * steps * u, atol=1e-30)
    # the update is at most lr x |m| / sqrt(v) <= lr / sqrt(1 - beta2) off by such a rounding per step
    lr, b2 = 1e-2, kw.get("betas", (0.9, 0.95))[1]
    torch.testing.assert_close(ga["master"], gb["master"], rtol=steps * u, atol=16 * steps * u * lr / (1 - b2) ** 0.5)
    ulp = {torch.float32: steps * u, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}[dtype]
    torch.testing.assert_close(ga["flat"].float(), gb["flat"].float(), rtol=ulp, atol=16 * steps * u * lr / (1 - b2) ** 0.5)


@pytest.mark.gpu
def test_state_that_is_not_aligned_takes_the_elementwise_loop(dccl_lib):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    a, b = (_train(_make(1, torch.bfloat16, [1000], general), 1) for general in (False, True))
    st = a.inner.state[a.groups[0]["master"]]
    for k in ("exp_avg", "exp_avg_sq"):                    # as after loading state that lies inside a larger buffer
        buf = torch.zeros(st[k].numel() + 1, device="cuda")
        buf[1:].copy_(st[k])
        st[k] = buf[1:]
    assert a._adamw_updates() is not None
    a, b = _train(a, 2), _train(b, 2)
    torch.testing.assert_close(a.groups[0]["master"], b.groups[0]["master"], rtol=3 * 2.0 ** -23, atol=1e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kw", [{}, {"betas": (0.0, 0.0), "eps": 0.0}, {"betas": (0.6, 0.999)}])
def test_infinities_nan_and_gradients_whose_squares_leave_the_range(dccl_lib, dtype, kw):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    vals = torch.tensor([float("inf"), float("-inf"), float("nan"), 2e19, -2e19, 1e20, 3e38, -3e38, 1.8e19, 1.9e19, 5e18, 1e-22, 1e-40, 0.0, 1.0], device="cuda")
    outs = []
    for general in (False, True):
        opt = _make(1, dtype, [vals.numel()], general, **kw)
        g = opt.groups[0]
        for sign in (0.0, 1.0, -1.0, 1.0):           # a plain step first
            g["grad"].zero_()
            if sign:
                g["grad"][:vals.numel()] = (sign * vals).to(dtype)
            opt.step()
        st = opt.inner.state[g["master"]]
        outs.append([t.detach().clone() for t in (g["master"], g["flat"], st["exp_avg"], st["exp_avg_sq"])])
    for x, y in zip(*outs):
        assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x.isinf(), y.isinf())
        fine = y.isfinite()
        # a few roundings per step, relative to gradients of both signs
        torch.testing.assert_close(x[fine].float(), y[fine].float(), rtol=2.0 ** -7 if x.dtype == torch.bfloat16 else 1e-5, atol=1e-7)


@pytest.mark.gpu
def test_two_slices_changed_options_and_loaded_state(dccl_lib):
    """One kernel per dtype; options changed between steps and state that went through state_dict are what the step uses."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")

    def make(general):
        torch.manual_seed(3)
        params = [torch.nn.Parameter(torch.randn(s, device="cuda").to(d)) for s, d in ((1001, torch.bfloat16), (77, torch.float32), (30, torch.bfloat16))]
        opt = zero.ShardedOptimizer(params, OneProcess(1), symmetric=False, lr=1e-2)
        if general:
            opt.inner.register_step_pre_hook(lambda *a: None)
        return opt

    a, b = _train(make(False), 2), _train(make(True), 2)
    for opt in (a, b):
        opt.inner.load_state_dict(opt.inner.state_dict())
        opt.inner.param_groups[0].update(lr=3e-3, weight_decay=0.5, eps=1e-4)
    assert len(a.groups) == 2 and a._adamw_updates() is not None
    a, b = _train(a, 2), _train(b, 2)
    for ga, gb in zip(a.groups, b.groups):
        torch.testing.assert_close(ga["master"], gb["master"], rtol=4 * 2.0 ** -23, atol=1e-7)
        assert float(a.inner.state[ga["master"]]["step"]) == 4


@pytest.mark.parametrize("kw,cls", [({"amsgrad": True}, torch.optim.AdamW), ({"maximize": True}, torch.optim.AdamW), ({}, torch.optim.Adam),
                                    ({"lr": torch.tensor(1e-2)}, torch.optim.AdamW), ({}, torch.optim.SGD), ({}, torch.optim.AdamW)])
def test_everything_else_stays_on_the_general_path(kw, cls):
    """Host tensors, with any options and optimizer. (What keeps tensors on a GPU from the kernel: further below.)"""
    opts = dict(kw)
    if cls is torch.optim.SGD:
        params = [torch.nn.Parameter(torch.randn(5))]
        opt = zero.ShardedOptimizer(params, OneProcess(1), cls, symmetric=False, lr=0.1)
    else:
        opt = _make(1, torch.float32, [5], False, device="cpu", cls=cls, **opts)
    before = opt.groups[0]["flat"].clone()
    _train(opt, 2)
    assert opt._adamw_updates() is None and not torch.equal(before, opt.groups[0]["flat"])


def _stepped(general, cls=torch.optim.AdamW, dtype=torch.float32, **kw):
    """One step done: the state exists, and is the same bits on every path, because the first step is torch's own."""
    return _train(_make(1, dtype, [1001], general, cls=cls, **kw), 1)


def _same_after_a_step(a, b):
    """One more step on both, and the same bits from it."""
    before = a.groups[0]["flat"].clone()
    for opt in (a, b):
        _train(opt, 1)
    for key in ("flat", "master"):
        assert torch.equal(a.groups[0][key], b.groups[0][key])
    assert not torch.equal(a.groups[0]["flat"], before)


@pytest.fixture
def cuda_lib(dccl_lib):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    assert _stepped(False)._adamw_updates() is not None        # what every case below changes one thing of


def test_a_function_put_in_place_of_the_class_step_or_around_it_is_noticed(monkeypatch):
    _make(1, torch.float32, [5], False, device="cpu")          # from the first object on, torch's base class wraps the step
    assert zero._step_is_torchs_own()
    stock = torch.optim.AdamW.step

    def step(self, *args):
        return stock(self, *args)

    for other in (step, functools.wraps(stock)(step), functools.partialmethod(stock), torch.optim.Optimizer.profile_hook_step(step)):
        monkeypatch.setattr(torch.optim.AdamW, "step", other)
        assert not zero._step_is_torchs_own()
    monkeypatch.setattr(torch.optim.AdamW, "step", stock)
    assert zero._step_is_torchs_own()


@pytest.mark.gpu
@pytest.mark.parametrize("wraps", [False, True])
def test_a_step_replaced_on_the_class_runs(cuda_lib, monkeypatch, wraps):
    a, b = _stepped(False), _stepped(True)
    stock, calls = torch.optim.AdamW.step, []

    def step(self, *args):
        calls.append(self)
        return stock(self, *args)

    monkeypatch.setattr(torch.optim.AdamW, "step", functools.wraps(stock)(step) if wraps else step)
    _same_after_a_step(a, b)
    assert calls == [a.inner, b.inner]


class SeesDispatch(TorchDispatchMode):
    """Counts what passes it."""
    seen = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen += 1
        return func(*args, **(kwargs or {}))


class SeesFunctions(TorchFunctionMode):
    seen = 0

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen += 1
        return func(*args, **(kwargs or {}))


def test_which_modes_count():
    assert not zero._a_mode_is_active()
    for mode in (SeesDispatch, SeesFunctions):
        with mode():
            assert zero._a_mode_is_active()
            with torch.device("cpu"):
                assert zero._a_mode_is_active()
        with torch.device("cpu"):
            assert not zero._a_mode_is_active()
            with mode():
                assert zero._a_mode_is_active()
    assert not zero._a_mode_is_active()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [SeesDispatch, SeesFunctions])
def test_an_active_mode_sees_the_operations_of_the_step(cuda_lib, mode):
    a, b = _stepped(False), _stepped(True)
    with mode() as m:
        a.step()
    assert m.seen > 3
    b.step()
    assert torch.equal(a.groups[0]["flat"], b.groups[0]["flat"])
    with torch.device("cuda"):                                  # a mode, too, but one that only places new tensors
        assert a._adamw_updates() is not None
        with mode():
            assert a._adamw_updates() is None


def test_ranges_are_entered_while_something_observes_them(tmp_path):
    assert not zero._observed()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert zero._observed()
    trace = torch.profiler.ExecutionTraceObserver()
    trace.register_callback(str(tmp_path / "trace.json"))
    trace.start()
    seen = zero._observed()
    trace.stop()
    trace.unregister_callback()
    assert seen and not zero._observed()


@pytest.mark.gpu
@pytest.mark.parametrize("observer", ["profiler", "execution trace"])
def test_the_profiler_range_of_the_step_is_there_on_both_paths(cuda_lib, monkeypatch, tmp_path, observer):
    for general in (False, True):
        opt, told = _stepped(general), []
        monkeypatch.setattr(opt.inner, "_optimizer_step_code", lambda: told.append(1), raising=False)
        if observer == "profiler":
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
                opt.step()
            ranges = [e for e in prof.events() if e.name == "Optimizer.step#AdamW.step"]
            assert len(ranges) == 1 and ranges[0].is_user_annotation
        else:
            path = str(tmp_path / ("%s.json" % general))
            trace = torch.profiler.ExecutionTraceObserver()
            trace.register_callback(path)
            trace.start()
            opt.step()
            trace.stop()
            trace.unregister_callback()
            assert "Optimizer.step#AdamW.step" in open(path).read()
        assert told == [1]


def _option(name, value):
    def change(opt, monkeypatch):
        opt.inner.param_groups[0][name] = value() if callable(value) else value
    return change


def _state(name, value):
    def change(opt, monkeypatch):
        st = opt.inner.state[opt.groups[0]["master"]]
        st[name] = value(st[name])
    return change


def _replaced_on_the_instance(opt, monkeypatch):
    opt.inner.step = functools.partial(type(opt.inner).step, opt.inner)


def _another_group(opt, monkeypatch):
    opt.inner.add_param_group({"params": [torch.nn.Parameter(torch.zeros(3, device="cuda"))]})


def _another_parameter(opt, monkeypatch):
    opt.inner.param_groups[0]["params"].append(torch.nn.Parameter(torch.zeros(3, device="cuda")))


def _hook(register):
    def change(opt, monkeypatch):
        monkeypatch.callbacks.append(register(opt.inner)(lambda *a: None))
    return change


def _between(x):
    return torch.stack([x, x], 1)[:, 0]                         # every second element of twice as many


@pytest.mark.gpu
@pytest.mark.parametrize("change", [
    _option("maximize", True), _option("decoupled_weight_decay", False), _option("lr", lambda: torch.tensor(1e-2)), _another_group, _another_parameter, _replaced_on_the_instance,
    _hook(lambda o: o.register_step_pre_hook), _hook(lambda o: o.register_step_post_hook),
    _hook(lambda o: register_optimizer_step_pre_hook), _hook(lambda o: register_optimizer_step_post_hook),
    _state("exp_avg", _between), _state("exp_avg_sq", _between),
], ids=["maximize", "coupled decay", "tensor lr", "two groups", "two parameters", "replaced step", "pre hook", "post hook", "global pre hook", "global post hook", "strided m", "strided v"])
def test_one_change_takes_the_general_path(cuda_lib, monkeypatch, change):
    monkeypatch.callbacks = []
    a, b = _stepped(False), _stepped(True)
    try:
        for opt in (a, b):
            change(opt, monkeypatch)
        assert a._adamw_updates() is None
        _same_after_a_step(a, b)
    finally:
        for c in monkeypatch.callbacks:
            c.remove()


@pytest.mark.gpu
@pytest.mark.parametrize("change", [
    # torch refuses some of these; the kernel must not get them before it does
    _option("amsgrad", True), _option("capturable", True), _option("differentiable", True), _option("fused", True), _option("weight_decay", lambda: torch.tensor(0.1)),
    _option("eps", lambda: torch.tensor(1e-8)), _option("betas", lambda: (torch.tensor(0.9), 0.95)), _option("betas", lambda: (0.9, torch.tensor(0.95))),
    _state("step", lambda x: x.cuda()), _state("step", float), _state("exp_avg", lambda x: x[:-1]), _state("exp_avg", lambda x: x.double()),
    _state("exp_avg", lambda x: None), _state("exp_avg_sq", lambda x: x.cpu()), _state("exp_avg_sq", lambda x: torch.nn.Parameter(x)),
], ids=["amsgrad", "capturable", "differentiable", "fused", "tensor decay", "tensor eps", "tensor beta 1", "tensor beta 2", "step on the GPU", "step a number", "m too short",
        "m in fp64", "no m", "v on the host", "v of a subclass"])
def test_options_and_state_the_kernel_does_not_take(cuda_lib, monkeypatch, change):
    opt = _stepped(False)
    change(opt, monkeypatch)
    assert opt._adamw_updates() is None


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [lambda s: s.double(), lambda s: s.reshape(1), lambda s: s.long(), lambda s: torch.nn.Parameter(s, requires_grad=False)],
                         ids=["fp64", "one element", "integer", "subclass"])
def test_step_counts_of_other_kinds_are_counted_in_place(cuda_lib, monkeypatch, kind):
    a, b = _stepped(False), _stepped(True)
    _state("step", kind)(a, monkeypatch)                        # torch's own step does not take all of these
    assert a._adamw_updates() is not None
    count = a.inner.state[a.groups[0]["master"]]["step"]
    version = count._version
    a, b = _train(a, 2), _train(b, 2)
    assert a.inner.state[a.groups[0]["master"]]["step"] is count and count.item() == 3 and count._version == version + 2
    torch.testing.assert_close(a.groups[0]["master"], b.groups[0]["master"], rtol=3 * 2.0 ** -23, atol=1e-7)


@pytest.mark.gpu
def test_a_step_count_that_torch_refuses_to_change(cuda_lib):
    opt = _stepped(False)
    st, before = opt.inner.state[opt.groups[0]["master"]], opt.groups[0]["flat"].clone()
    with torch.inference_mode():
        st["step"] = st["step"].clone()
    with pytest.raises(RuntimeError, match="[Ii]nference"):
        opt.step()
    assert torch.equal(opt.groups[0]["flat"], before)


@pytest.mark.gpu
@pytest.mark.parametrize("count", [-1.0, -0.5, -3.0, float("-inf")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_step_counts_below_zero_are_torchs_to_report(cuda_lib, monkeypatch, count, dtype):
    a, b = _stepped(False), _stepped(True)
    for opt in (a, b):
        _state("step", lambda s: torch.tensor(count, dtype=dtype))(opt, monkeypatch)
    assert a._adamw_updates() is None
    if count == -1:
        for opt in (a, b):
            with pytest.raises(ZeroDivisionError):
                opt.step()
        assert torch.equal(a.groups[0]["flat"], b.groups[0]["flat"]) and torch.isfinite(a.groups[0]["flat"]).all()


@pytest.mark.gpu
def test_what_a_step_changes_is_a_new_version(cuda_lib):
    opt = _stepped(False)
    g, st = opt.groups[0], opt.inner.state[opt.groups[0]["master"]]
    changed = (g["master"], g["master"].grad, st["exp_avg"], st["exp_avg_sq"], st["step"], g["flat"])
    before = [x._version for x in changed] + [g["grad"]._version]
    opt.step()
    assert [x._version for x in changed] + [g["grad"]._version] == [v + 1 for v in before[:-1]] + before[-1:]


@pytest.mark.gpu
@pytest.mark.parametrize("betas,taken", [([0.9, 0.95], True), ((0, 0.95), True), ((1.0, 0.95), False), ((0.9, 1.0), False), ((-0.1, 0.95), False),
                                         ((0.9, float("nan")), False), ((0.9,), False), ((0.9, "0.95"), False)])
def test_betas_the_kernel_takes(cuda_lib, betas, taken):
    opt = _stepped(False)
    opt.inner.param_groups[0]["betas"] = betas
    assert (opt._adamw_updates() is not None) == taken


def test_without_the_extension_torch_steps(monkeypatch):
    def broken():
        raise RuntimeError("no compiler")

    monkeypatch.setattr(zero, "_native", None)
    monkeypatch.setattr(zero.backend_build, "load", broken)
    with pytest.warns(UserWarning, match="no compiler"):
        assert zero._native_step() == ()
    assert zero._native_step() == ()                            # said once


@pytest.mark.gpu
@pytest.mark.parametrize("name,value", [("amsgrad", 0), ("maximize", np.False_), ("fused", 0), ("decoupled_weight_decay", 1), ("betas", np.array([0.9, 0.95])),
                                        ("betas", collections.deque([0.9, 0.95])), ("betas", collections.UserList([0.9, 0.95])), ("lr", np.float64(1e-2)), ("eps", 0)])
def test_options_that_python_takes_for_plain_ones(cuda_lib, monkeypatch, name, value):
    a, b = _stepped(False), _stepped(False)
    _option(name, lambda: value)(a, monkeypatch)
    if name == "eps":
        b.inner.param_groups[0]["eps"] = 0.0
    assert a._adamw_updates() is not None
    _same_after_a_step(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("name,value", [("amsgrad", 1), ("maximize", torch.ones(2, dtype=torch.bool)), ("decoupled_weight_decay", 0), ("betas", np.array([0.9])),
                                        ("betas", 0.9), ("betas", np.array([0.9, 0.95], dtype=np.float32)), ("betas", collections.deque([0.9, 0.95, 0.99]))])
def test_options_that_python_takes_for_others(cuda_lib, monkeypatch, name, value):
    opt = _stepped(False)
    _option(name, lambda: value)(opt, monkeypatch)
    assert opt._adamw_updates() is None


def test_the_entry_point_is_declared_once(dccl_lib, monkeypatch):
    """By the header: the extension, which calls it by address, is older than a changed one, and ctypes has the same arguments."""
    if not hasattr(dccl_lib, "dccl_adamw_flat"):
        pytest.skip("a host-only library")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    header = os.path.join(root, "csrc", "kernels", "adamw.hpp")
    kinds = {"int": ctypes.c_int, "size_t": ctypes.c_size_t, "double": ctypes.c_double}
    arguments = re.search(r"int dccl_adamw_flat\((.*?)\);", open(header).read(), re.S).group(1).split(",")
    assert dccl_lib.dccl_adamw_flat.argtypes == [ctypes.c_void_p if "*" in a else kinds[a.split()[0]] for a in arguments]
    for name in ("kernels/adamw.cu", "torch/adamw_step.cpp"):
        assert "adamw.hpp\"" in open(os.path.join(root, "csrc", name)).read()
    zero.backend_build.build()
    stock = os.path.getmtime
    monkeypatch.setattr(os.path, "getmtime", lambda f: 1e12 if os.path.realpath(f) == os.path.realpath(header) else stock(f))
    assert zero.backend_build.needs_build()


def test_the_extension_is_loaded_without_a_compiler_or_not_at_all(monkeypatch, tmp_path):
    """What an optimizer does while it is made: no rank of a job compiles for a minute there."""
    monkeypatch.setattr(zero.backend_build, "_module", None)
    monkeypatch.setattr(zero.backend_build, "OUT", str(tmp_path / "missing.so"))
    monkeypatch.setattr(zero.backend_build.subprocess, "run", lambda *a, **kw: pytest.fail("a compiler is run"))
    with pytest.raises(ImportError, match="missing.so"):
        zero.backend_build.load()
    monkeypatch.setattr(zero, "_native", None)
    with pytest.warns(UserWarning, match="missing.so"):
        assert zero._native_step() == ()


@pytest.fixture
def no_extension(cuda_lib, monkeypatch):
    def missing():
        raise ImportError("no extension")

    monkeypatch.setattr(zero, "_native", None)
    monkeypatch.setattr(zero.backend_build, "load", missing)


@pytest.mark.gpu
@pytest.mark.parametrize("world", [1, 2])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_an_optimizer_without_the_extension_steps_as_one_kernel(dccl_lib, no_extension, monkeypatch, world, dtype):
    outs = []
    for extension in (False, True):
        if extension:
            monkeypatch.undo()
            opt = _make(world, dtype, [2049, 7], False)
        else:
            with pytest.warns(UserWarning, match="no extension"):
                opt = _make(world, dtype, [2049, 7], False)
        _train(opt, 1)
        general = []
        opt.inner._optimizer_step_code = lambda: general.append(opt._adamw_updates())
        _train(opt, 3)
        assert len(general) == 3 and None not in general and (zero._native != ()) == extension
        g = opt.groups[0]
        st = opt.inner.state[g["master"]]
        outs.append([g["master"], g["master"].grad, g["flat"], st["exp_avg"], st["exp_avg_sq"], st["step"]])
        assert [x._version for x in outs[-1]] == [x._version for x in outs[0]]
    assert all(torch.equal(x, y) for x, y in zip(*outs))


@pytest.mark.gpu
@pytest.mark.parametrize("change", [
    _option("lr", 1), _option("amsgrad", 0), _option("amsgrad", 1), _option("maximize", torch.ones(2, dtype=torch.bool)), _option("capturable", True),
    _option("differentiable", True), _option("fused", True), _option("decoupled_weight_decay", 0), _option("betas", (1.0, 0.95)), _option("betas", (0.9, float("nan"))),
    _option("betas", (0.9,)), _option("betas", 0.9), _option("betas", (0.9, "0.95")), _option("betas", np.array([0.9, 0.95])), _option("betas", (0, 0.95)),
    _option("eps", 10 ** 400), _option("eps", lambda: torch.tensor(1e-8)), _option("weight_decay", None),
    _state("step", float), _state("step", lambda x: x.cuda()), _state("step", lambda x: -x - 0.5), _state("step", lambda x: x.double()), _state("step", lambda x: x.repeat(2)),
    _state("step", lambda x: x.to(torch.complex64)), _state("step", lambda x: x * float("nan")),
    _state("exp_avg", lambda x: x[:-1]), _state("exp_avg", lambda x: x.double()), _state("exp_avg", lambda x: None), _state("exp_avg", _between),
    _state("exp_avg_sq", lambda x: x.cpu()), _state("exp_avg_sq", lambda x: torch.nn.Parameter(x)),
])
def test_both_hosts_take_the_same_slices(cuda_lib, monkeypatch, change):
    opt = _stepped(False)
    change(opt, monkeypatch)
    native = opt._adamw_updates() is not None
    monkeypatch.setattr(zero, "_native", ())
    assert (opt._adamw_updates() is not None) == native


@pytest.mark.gpu
def test_optimizers_dtypes_and_surroundings_the_kernel_does_not_take(cuda_lib, monkeypatch):
    assert _stepped(False, cls=torch.optim.Adam)._adamw_updates() is None
    assert _stepped(False, cls=type("Derived", (torch.optim.AdamW,), {}))._adamw_updates() is None
    assert _stepped(False, dtype=torch.float64)._adamw_updates() is None
    assert _make(1, torch.float32, [5], False)._adamw_updates() is None            # no state yet
    opt = _stepped(False)
    opt.groups[0]["master"].grad = None
    assert opt._adamw_updates() is None
    opt = _stepped(False)
    other = opt.groups[0]["master"].detach().clone().requires_grad_(True)
    other.grad = torch.zeros_like(other)
    opt.inner.state[other] = opt.inner.state[opt.groups[0]["master"]]
    opt.inner.param_groups[0]["params"][0] = other
    assert opt._adamw_updates() is None
    opt = _stepped(False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = opt._adamw_updates()
        torch.zeros(1, device="cuda")
    assert captured is None and opt._adamw_updates() is not None
    monkeypatch.setattr(torch.compiler, "is_compiling", lambda: True)
    assert opt._adamw_updates() is None


@pytest.mark.gpu
def test_the_update_is_ordered_on_a_side_stream(cuda_lib):
    a, b = _stepped(False), _stepped(True)
    grad = torch.randn(a.groups[0]["grad"].numel(), device="cuda")
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(3):
            torch.cuda._sleep(2000000)                          # about a millisecond: a launch elsewhere would come first
            a.groups[0]["grad"].copy_(grad)
            a.step()
            a.groups[0]["grad"].fill_(float("nan"))
    side.synchronize()
    for _ in range(3):
        b.groups[0]["grad"].copy_(grad)
        b.step()
    torch.testing.assert_close(a.groups[0]["flat"], b.groups[0]["flat"], rtol=4 * 2.0 ** -23, atol=1e-7)


@pytest.mark.gpu
def test_a_scheduler_made_late_sees_the_next_step(cuda_lib):
    """Its first step warns unless the optimizer has stepped since it was made, on either path."""
    for general in (False, True):
        opt = _stepped(general)
        sched = torch.optim.lr_scheduler.LambdaLR(opt.inner, lambda t: 0.5 ** t)
        with warnings.catch_warnings():
            warnings.simplefilter("error")
            _train(opt, 1)
            sched.step()
        assert opt.inner.param_groups[0]["lr"] == 0.5e-2
