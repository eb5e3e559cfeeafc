"""Builds ``libtuisko_sm100.so`` in-tree with nvcc for sm_100a (the only target), and the CPython
binding of its launches (``_native.<torch version><extension suffix>``) with the host compiler."""
from __future__ import annotations

import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libtuisko_sm100.so")
BINDING_SOURCE = os.path.join(CSRC, "binding.cpp")
SOURCES = ["norm_quant.cu", "fp8_proj.cu", "fp8_pair.cu", "fp8_mlp.cu", "gdn.cu", "materialize.cu", "nvfp4.cu", "nvfp4_pair.cu", "pair_gemm.cu", "peer_reduce.cu", "sampler.cu", "ops.cu", "static_entry.cu"]
HEADERS = ["common.cuh", "ptx.cuh", "kernels.h", "ops.hpp", "../../include/tuisko_sm100.h"]


def nvcc_path() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; tuisko-kernels-sm100 has no prebuilt or CPU fallback")


def is_stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def binding_path() -> str:
    """Named after what it is compiled against -- torch's C++ ABI and the interpreter's -- so that a copy
    built for another of either is not taken for this one's."""
    import torch

    return os.path.join(HERE, "_native.%s%s" % (torch.__version__, sysconfig.get_config_var("EXT_SUFFIX")))


def binding_is_stale() -> bool:
    path = binding_path()
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    deps = [BINDING_SOURCE, os.path.abspath(os.path.join(CSRC, "../../include/tuisko_sm100.h")),
            importlib.util.find_spec("torch").origin]  # compiled against this torch's headers
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles the library when it is absent or older than its sources.  Several processes may
    call this at once (one rank per GPU): an exclusive file lock lets one of them compile, into a
    temporary file that is renamed into place, and the others then find the library fresh."""
    return _build_locked(LIB, is_stale, _compile, force, verbose)


def build_binding(force: bool = False, verbose: bool = False) -> str:
    """The same for the launch binding."""
    return _build_locked(binding_path(), binding_is_stale, _compile_binding, force, verbose)


def _build_locked(path, stale, compile_it, force, verbose) -> str:
    if not force and not stale():
        return path
    import fcntl

    with open(path + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not stale():  # another process built it while this one waited
                return path
            return compile_it(verbose)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def _compile(verbose: bool) -> str:
    """TK100_EXPERIMENT=1 in the environment of the build adds -DTK100_EXPERIMENT: the library
    then honours the TK100_DEBUG performance-experiment bits (which make results wrong); the
    default build has no such code."""
    tmp = "%s.%d.tmp" % (LIB, os.getpid())
    cmd = [
        nvcc_path(), "-std=c++17", "-O3", "-lineinfo",
        "-gencode", "arch=compute_100a,code=sm_100a",
        "-Xcompiler", "-fPIC,-fvisibility=hidden", "-shared",
        "-Xptxas", "-v" if verbose else "-warn-spills",
        "-o", tmp,
    ] + (["-DTK100_EXPERIMENT"] if os.environ.get("TK100_EXPERIMENT") == "1" else []) \
      + [os.path.join(CSRC, s) for s in SOURCES] + ["-lcudart_static", "-ldl", "-lrt", "-lpthread"]
    # the image exports CC/CXX pointing at a private gcc; nvcc wants the system one
    if os.path.exists("/usr/bin/g++"):
        cmd[1:1] = ["-ccbin", "/usr/bin/g++"]
    return _run(cmd, tmp, LIB, verbose)


def _compile_binding(verbose: bool) -> str:
    path = binding_path()
    tmp = "%s.%d.tmp" % (path, os.getpid())
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc_path())))
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else os.environ.get("CXX", "g++")
    cmd = [cxx, "-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden", "-shared", "-o", tmp, BINDING_SOURCE]
    cmd += ["-I" + d for d in (os.path.join(torch_dir, "include"),
                               os.path.join(torch_dir, "include/torch/csrc/api/include"),
                               sysconfig.get_paths()["include"], os.path.join(cuda, "include"))]
    cmd += ["-L" + os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    return _run(cmd, tmp, path, verbose)


def _run(cmd, tmp, path, verbose) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        if os.path.exists(tmp):
            os.unlink(tmp)
        raise RuntimeError("building %s failed" % os.path.basename(path))
    os.replace(tmp, path)  # atomic: a concurrent loader sees the old file or the new one, whole
    return path


if __name__ == "__main__":
    print(build(force=True, verbose="-v" in sys.argv))
    print(build_binding(force=True, verbose="-v" in sys.argv))
