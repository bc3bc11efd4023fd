"""Builds the PyTorch extension (csrc/torch: the process-group backend and the host side of the AdamW update) in-tree, next to
libdccl.so, and loads it.

The extension only uses the library's public C++ API and libtorch; it is compiled with the system
C++ compiler against the headers of the installed torch and linked to ``dccl_b200/lib/libdccl.so``
by relative rpath, so the built file can be moved with the package. Its name carries the versions of torch and of Python whose
inline code it holds: after either is replaced, it is a missing file and not one that reads objects of another layout.
"""
import fcntl
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
_PKG = os.path.dirname(_HERE)
_ROOT = os.path.dirname(_PKG)
SRC_DIR = os.path.join(_ROOT, "csrc", "torch")
SRCS = [os.path.join(SRC_DIR, name) for name in ("pg_dccl.cpp", "adamw_step.cpp")]
HEADERS = [os.path.join(SRC_DIR, "adamw_step.hpp"), os.path.join(_ROOT, "csrc", "kernels", "adamw.hpp"), os.path.join(_ROOT, "include", "dccl", "dccl.hpp")]
OUT = os.path.join(_PKG, "lib", "_dccl_torch-%s-torch%s.so" % (sys.implementation.cache_tag, torch.__version__))


def needs_build():
    if not os.path.exists(OUT):
        return True
    # a package that came without its sources is as new as it gets
    return any(os.path.exists(f) and os.path.getmtime(OUT) < os.path.getmtime(f) for f in SRCS + HEADERS)


def build(force=False, verbose=False):
    """Compiles the extension unless it is up to date. Of several ranks one compiles and the others wait for its file."""
    if not force and not needs_build():
        return OUT
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    with open(OUT + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)        # given back by the system when its holders have ended: this process and the compiler
        if force or needs_build():
            _compile(lock, verbose)
    return OUT


def _compile(lock, verbose):
    from torch.utils import cpp_extension
    from .._lib import LIB_PATH, lib
    lib()   # makes sure libdccl.so exists
    # a compiler that links libstdc++ dynamically, like torch itself does
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else (shutil.which("g++") or "c++")
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    incs = cpp_extension.include_paths(device_type="cuda")
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    part = OUT + ".part"                        # one name: what a killed compiler left is written over by the next
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", *SRCS, "-o", part,
           "-DTORCH_EXTENSION_NAME=_dccl_torch", "-DTORCH_API_INCLUDE_EXTENSION_H", "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
           "-I" + os.path.join(_ROOT, "include"), "-I" + os.path.join(cuda_home, "include"), "-I" + sysconfig.get_paths()["include"]]
    cmd += ["-I" + p for p in incs]
    cmd += ["-L" + tlib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
            "-L" + os.path.dirname(LIB_PATH), "-ldccl", "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + tlib, "-Wno-attributes", "-Wno-interference-size"]
    res = subprocess.run(cmd, capture_output=True, text=True, pass_fds=(lock.fileno(),))
    if res.returncode != 0:
        raise RuntimeError("building the torch backend failed:\n" + " ".join(cmd) + "\n" + res.stderr[-6000:])
    os.replace(part, OUT)
    if verbose:
        print(res.stderr, file=sys.stderr)


_module = None


def load(compile=False):
    """The extension module. A file that is missing or older than its sources is compiled first, or an ImportError."""
    global _module
    if _module is None:
        if compile:
            build()
        elif needs_build():
            raise ImportError("%s is missing or older than its sources (python -m dccl_b200.parallel.backend_build builds it)" % OUT)
        spec = importlib.util.spec_from_file_location("_dccl_torch", OUT)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        _module = module
    return _module


if __name__ == "__main__":
    print(build(force=True, verbose=True))
