"""Data parallelism with the optimizer state split over the ranks (ZeRO stage 1 / 2 style).

The gradient all-reduce of plain data parallelism is a reduce-scatter followed by an all-gather (the
original builds its ring all-reduce exactly so, reference src/core/all_reduce_ring.cpp:8-79). Here the
optimizer step sits between the two halves: every rank reduces only its 1/world slice of the flat gradient,
updates the matching slice of the parameters with its own slice of the optimizer state, and the updated
slices are gathered. Communication volume is that of one all-reduce; optimizer memory and update work
drop to 1/world per rank.

    params -> one flat buffer per dtype (padded to world x 16 bytes), ``p.data`` and ``p.grad`` are views
    step:    reduce_scatter(avg) flat_grad -> grad slice (fp32 copy when the parameters are 16-bit)
             inner optimizer on the master slice (fp32); AdamW runs as one kernel together with the casts on either side
             all_gather the updated slice (cast back) into the flat parameter buffer

With ``comm.world == 1`` this is the inner optimizer on a flat buffer. CPU tensors use the host path, CUDA
tensors the device kernels on the current stream; on GPUs with NVSwitch multicast the flat buffers live in
symmetric memory (``symmetric=True``), so that both collectives run zero-copy through the switch. Call
``close()`` before the communicator is finalized to give that memory back.
"""
import ctypes
import math
import os
import warnings

import torch
import torch.optim.adam as _adam
import torch.optim.optimizer as _optimizer
from torch.utils._device import DeviceContext

from .._lib import lib
from ..comm import DcclError, current_stream_handle, dtype_of
from . import backend_build

_FUSED_DTYPES = (torch.bfloat16, torch.float16, torch.float32)
_IN_OPTIMIZER, _IN_ADAM = vars(_optimizer), vars(_adam)
_enter_range, _exit_range = torch._C._autograd._record_function_with_args_enter, torch._C._autograd._record_function_with_args_exit


def _observer_query():
    """hasCallbacks of torch's C++ API (ATen/record_function.h): whether anything looks at ranges, be it the profiler or an
    observer without it. A torch that does not export it is taken to be observed always."""
    try:
        f = ctypes.PyDLL(os.path.join(os.path.dirname(torch.__file__), "lib", "libtorch_cpu.so"))._ZN2at12hasCallbacksEv
    except (OSError, AttributeError):
        return lambda: True
    f.restype, f.argtypes = ctypes.c_bool, []
    return f


_observed = _observer_query()

_native = None


def _native_step():
    """(check, update, address of the launch) of the host side of the one-kernel update (csrc/torch/adamw_step.cpp), or () where
    the extension that holds it has not been built or cannot be loaded: _adamw_ready and _adamw_update do the same then."""
    global _native
    if _native is None:
        try:
            ext = backend_build.load()
            _native = ext.adamw_ready, ext.adamw_update, ctypes.cast(lib().dccl_adamw_flat, ctypes.c_void_p).value
        except (ImportError, OSError, RuntimeError, AttributeError) as e:
            warnings.warn("dccl_b200: the host side of sharded AdamW steps runs in Python, which counts for small models: %s" % e)
            _native = ()
    return _native


def _adamw_ready(o, st, p, p_grad, grad, n):
    """adamw_ready of csrc/torch/adamw_step.cpp, with the same answers."""
    try:
        if o["amsgrad"] or o["maximize"] or o["capturable"] or o["differentiable"] or o["fused"] or not o.get("decoupled_weight_decay", True):
            return False
        lr, decay, eps, (b1, b2) = o["lr"], o["weight_decay"], o["eps"], o["betas"]
        for x in (lr, decay, eps, b1, b2):
            if not isinstance(x, (int, float)):
                return False
        if not (0 <= b1 < 1 and 0 <= b2 < 1):
            return False
        lr + decay + eps + 0.0
    except Exception:       # missing, without a truth value, no pair, an integer beyond any float: torch's step reports it
        return False
    count, device = st.get("step"), p.get_device()
    if device < 0 or type(grad) is not torch.Tensor or grad.dtype not in _FUSED_DTYPES or not isinstance(count, torch.Tensor) or count.is_cuda:
        return False
    # below zero the bias corrections divide by zero or have no square root, which torch's step reports
    if count.numel() != 1 or count.is_complex() or not count.item() >= 0:
        return False
    for t in (p, p_grad, st.get("exp_avg"), st.get("exp_avg_sq")):
        if type(t) is not torch.Tensor or t.dtype is not torch.float32 or t.get_device() != device or t.numel() != n or not t.is_contiguous():
            return False
    return not torch.cuda.is_current_stream_capturing()


def _adamw_update(_, o, st, p, p_grad, grad, out, n):
    """adamw_update of csrc/torch/adamw_step.cpp. From Python a step of 0.4 M parameters takes 12.8 us, from the extension 5.6."""
    device, m, v = p.get_device(), st["exp_avg"], st["exp_avg_sq"]
    count, lr, (b1, b2) = st["step"], o["lr"], o["betas"]
    t = count.item() + 1
    count.fill_(t)
    rc = lib().dccl_adamw_flat(device, dtype_of(grad), n, p.data_ptr(), p_grad.data_ptr(), m.data_ptr(), v.data_ptr(), grad.data_ptr(), out.data_ptr(),
                               1 - lr * o["weight_decay"], 1 - b1, b2, 1 - b2, lr / (1 - b1 ** t), math.sqrt(1 - b2 ** t), o["eps"],
                               current_stream_handle(device))
    if rc == 0:
        torch.autograd.graph.increment_version((p, p_grad, m, v, out))
    return rc


_IN_PYTHON = _adamw_ready, _adamw_update, None


def _step_is_torchs_own():
    """Whether AdamW's class still has the step that torch wrote, under nothing but the wrappers that torch's base class puts
    around it: a function of another module in its place, or around it, has to run."""
    try:
        f = torch.optim.AdamW.step
        while f.__globals__ is _IN_OPTIMIZER:
            f = f.__wrapped__
        return f.__globals__ is _IN_ADAM
    except AttributeError:
        return False


def _a_mode_is_active():
    """Whether a mode would see torch's calls: any, except the one behind ``torch.device`` and the default device, which only
    places new tensors."""
    if torch._C._len_torch_dispatch_stack():
        return True
    n = torch._C._len_torch_function_stack()
    return n > 0 and any(type(torch._C._get_function_stack_at(i)) is not DeviceContext for i in range(n))


class ShardedOptimizer:
    """optimizer_cls(params, **kwargs) is built over ONE tensor per dtype: this rank's fp32 master slice."""

    def __init__(self, params, comm, optimizer_cls=torch.optim.AdamW, symmetric=True, **kwargs):
        self.comm = comm
        self._sym = []
        params = [p for p in params if p.requires_grad]
        if not params:
            raise ValueError("no trainable parameters")
        n, r = comm.world, comm.rank
        self.groups = []
        by_dtype = {}
        for p in params:
            by_dtype.setdefault((p.dtype, p.device), []).append(p)
        masters = []
        for (dtype, device), plist in by_dtype.items():
            itemsize = torch.empty((), dtype=dtype).element_size()
            align = 16 // itemsize
            offs, total = [], 0
            for p in plist:
                offs.append(total)
                total += -(-p.numel() // align) * align            # every view starts 16-byte aligned
            per = -(-total // (n * align)) * align                  # slice length, a whole number of 16-byte vectors
            if symmetric and device.type == "cuda" and n > 1 and comm.has_multicast:
                flat = comm.symmetric_empty(per * n, dtype, device.index).zero_()
                grad = comm.symmetric_empty(per * n, dtype, device.index).zero_()
                self._sym += [flat, grad]
            else:
                flat = torch.zeros(per * n, dtype=dtype, device=device)
                grad = torch.zeros(per * n, dtype=dtype, device=device)
            for p, off in zip(plist, offs):
                flat[off:off + p.numel()].copy_(p.data.reshape(-1))
                p.data = flat[off:off + p.numel()].view_as(p)
                p.grad = grad[off:off + p.numel()].view_as(p)
            master = flat[r * per:(r + 1) * per].detach().clone().float().requires_grad_(True)
            master.grad = torch.zeros_like(master)
            masters.append(master)
            self.groups.append({"flat": flat, "grad": grad, "per": per, "master": master, "params": plist,
                                "grad_slice": torch.empty(per, dtype=dtype, device=device),
                                "out_slice": torch.empty(per, dtype=dtype, device=device)})
        self.inner = optimizer_cls(masters, **kwargs)
        if optimizer_cls is torch.optim.AdamW and any(m.is_cuda for m in masters):
            _native_step()

    def zero_grad(self):
        for g in self.groups:
            g["grad"].zero_()

    def step(self):
        comm, n = self.comm, self.comm.world
        if n > 1:
            for g in self.groups:
                comm.reduce_scatter(g["grad"], g["grad_slice"], op="avg")
        updates = self._adamw_updates()
        if updates is not None:
            self._adamw_range(updates)
        else:
            for g in self.groups:
                g["master"].grad.copy_(g["grad_slice"] if n > 1 else g["grad"])
            self.inner.step()
            for g in self.groups:
                (g["out_slice"] if n > 1 else g["flat"]).copy_(g["master"].detach())
        if n > 1:
            for g in self.groups:
                comm.all_gather(g["out_slice"], g["flat"])

    def _adamw_updates(self):
        """(group, options, state) of every slice when one kernel per slice can do what ``inner.step()`` and the casts around
        it do: plain AdamW on CUDA, past its first step (which makes the state), with nothing hooked into the step that
        would have to see the gradient before or the result in between. None: the general path, which also reports
        whatever is wrong with the state."""
        inner = self.inner
        if type(inner) is not torch.optim.AdamW or not _step_is_torchs_own() or torch.compiler.is_compiling():
            return None
        if _a_mode_is_active():
            return None
        if (inner._optimizer_step_pre_hooks or inner._optimizer_step_post_hooks or _optimizer._global_optimizer_pre_hooks
                or _optimizer._global_optimizer_post_hooks):
            return None
        # a learning-rate scheduler wraps the step of its optimizer to see that it ran; any other replacement has to run
        step = inner.__dict__.get("step")
        if step is not None and not (getattr(step, "_wrapped_by_lr_sched", False) and getattr(step, "__wrapped__", None) is type(inner).step):
            return None
        if len(inner.param_groups) != 1 or len(inner.param_groups[0]["params"]) != len(self.groups):
            return None
        if not self.groups[0]["master"].is_cuda:
            return None
        ready, o, updates = (_native_step() or _IN_PYTHON)[0], inner.param_groups[0], []
        for g, p in zip(self.groups, o["params"]):
            # options of plain AdamW, state on the GPU as the kernel reads it, and no capture
            st = inner.state.get(p)
            if p is not g["master"] or not st or not ready(o, st, p, p.grad, g["grad"], g["per"]):
                return None
            updates.append((g, o, st))
        if step is not None:
            inner._opt_called = True
        return updates

    def _adamw_range(self, updates):
        """The updates, where torch's optimizers show their step: inside the range that the profiler and other observers know
        it by, with the call at its end through which the profiler finds the optimizer. An unobserved range costs a step
        2.0 us on top of 5.6 and is left out."""
        entered = _enter_range("Optimizer.step#AdamW.step") if _observed() else None
        try:
            for u in updates:
                self._adamw(*u)
            self.inner._optimizer_step_code()
        finally:
            if entered is not None:
                _exit_range(entered)

    def _adamw(self, g, o, st):
        p = g["master"]
        grad, out = (g["grad_slice"], g["out_slice"]) if self.comm.world > 1 else (g["grad"], g["flat"])
        _, update, launch = _native or _IN_PYTHON
        if update(launch, o, st, p, p.grad, grad, out, g["per"]) != 0:
            raise DcclError(1, "AdamW update")

    def close(self):
        """Give symmetric buffers back (collective). The parameters keep their values in ordinary memory."""
        if not self._sym:
            return
        torch.cuda.synchronize()
        for g in self.groups:
            keep = g["flat"].clone()
            off = 0
            for p in g["params"]:
                # same layout as in __init__: every view starts 16-byte aligned
                align = 16 // keep.element_size()
                p.data = keep[off:off + p.numel()].view_as(p)
                p.grad = None
                off += -(-p.numel() // align) * align
            g["flat"], g["grad"] = keep, torch.zeros_like(keep)
        for t in self._sym:
            self.comm.free_symmetric(t)
        self._sym = []

    def state_bytes(self):
        """Bytes of optimizer state held by this rank (for reports and tests)."""
        total = 0
        for st in self.inner.state.values():
            for v in st.values():
                if torch.is_tensor(v):
                    total += v.numel() * v.element_size()
        return total
