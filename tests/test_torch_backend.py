"""torch.distributed backend "dccl": every collective against values computed from the ranks' seeds,
DistributedDataParallel gradients against a serial reference. CPU tensors here; CUDA tensors in the
gpu-marked tests."""
import importlib.util
import os
import subprocess
import threading
import time
from concurrent.futures import ThreadPoolExecutor

import pytest

from conftest import gpu_count
from dccl_b200.parallel import backend_build
from dccl_b200.utils.launch import python_ranks

HERE = os.path.dirname(os.path.abspath(__file__))
WORKER = os.path.join(HERE, "workers", "torch_worker.py")


def run(world, args, gpus=False, timeout=600):
    res = python_ranks(WORKER, args, world, timeout=timeout, gpus=gpus)
    for r, p in enumerate(res):
        assert p.returncode == 0, "rank %d:\n%s\n%s" % (r, p.stdout[-2000:], p.stderr[-3000:])
        assert p.stdout.strip().endswith("OK")


def test_an_extension_of_another_torch_is_not_loaded(monkeypatch):
    backend_build.build()
    assert not backend_build.needs_build()
    monkeypatch.setattr(backend_build.torch, "__version__", "1.0.0")
    spec = importlib.util.spec_from_file_location("backend_build_of_another_torch", backend_build.__file__)
    other = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(other)
    assert other.needs_build()
    with pytest.raises(ImportError):
        other.load()


@pytest.mark.parametrize("force", [False, True])
def test_ranks_that_find_no_extension_compile_it_one_at_a_time(monkeypatch, tmp_path, force):
    out, running, compiled = str(tmp_path / "lib" / "extension.so"), threading.Lock(), []

    def compiler(cmd, **kw):
        assert running.acquire(blocking=False), "two compilers at a time"
        time.sleep(0.2)
        path = cmd[cmd.index("-o") + 1]
        with open(path, "w") as f:
            f.write("complete")
        compiled.append(path)
        running.release()
        return subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(backend_build, "OUT", out)
    monkeypatch.setattr(backend_build.subprocess, "run", compiler)
    with ThreadPoolExecutor(4) as ranks:
        assert [f.result() for f in [ranks.submit(backend_build.build, force) for _ in range(4)]] == [out] * 4
    assert len(compiled) == (4 if force else 1) and out not in compiled
    assert open(out).read() == "complete" and not [p for p in compiled if os.path.exists(p)]


def test_what_a_killed_compiler_leaves_does_not_pile_up(monkeypatch, tmp_path):
    monkeypatch.setattr(backend_build, "OUT", str(tmp_path / "extension.so"))
    left = set()
    for pid in (11, 12, 13):
        monkeypatch.setattr(backend_build.os, "getpid", lambda: pid)
        monkeypatch.setattr(backend_build.subprocess, "run", lambda cmd, **kw: (left.add(cmd[cmd.index("-o") + 1]), 1 / 0))
        with pytest.raises(ZeroDivisionError):
            backend_build.build()
    assert len(left) == 1


@pytest.mark.parametrize("world", [2, 4])
def test_collectives_and_ddp_on_cpu_tensors(world):
    run(world, ["--ddp", "--extra"])


@pytest.mark.gpu
@pytest.mark.skipif(gpu_count() < 2, reason="needs two GPUs")
def test_collectives_and_ddp_on_cuda_tensors():
    run(min(gpu_count(), 8), ["--cuda", "--ddp"], gpus=True)


@pytest.mark.gpu
def test_single_gpu_process_group():
    run(1, ["--cuda", "--ddp"], gpus=True)


@pytest.mark.gpu
@pytest.mark.skipif(gpu_count() < 2, reason="needs two GPUs")
def test_all_to_all_gather_scatter_batches_objects_subgroups_on_cuda_tensors():
    run(min(gpu_count(), 8), ["--cuda", "--extra"], gpus=True)
