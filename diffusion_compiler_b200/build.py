"""Builds libdifb200.so (sm_100a only) in-tree with nvcc.

    python -m diffusion_compiler_b200.build [--force]

The shared library carries every CUDA kernel, the device-resident C entry points
(include/difb200/difb200.h) and the reference-compatible backend plugin entry points
(include/difb200/abi.h). nvcc cross-compiles without a GPU. Beside it stands _torch_calls.so, the binding
that ops.py calls it through on torch tensors.
"""
from __future__ import annotations

import importlib.metadata
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(HERE, "_obj")
LIB_PATH = os.path.join(HERE, "libdifb200.so")
CALLS_SOURCE = os.path.join(HERE, "binding", "torch_calls.cpp")
CALLS_PATH = os.path.join(HERE, "_torch_calls.so")
CALLS_STAMP = os.path.join(OBJ_DIR, "torch_calls.stamp")  # what _torch_calls.so was built for

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
    "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall",
]


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp")))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = os.environ.get("NVCC", "nvcc")
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    inc = os.path.join(ROOT, "include", "difb200")
    headers += [os.path.join(inc, f) for f in os.listdir(inc)]
    jobs = []
    objs = []
    for src in _sources():
        obj = os.path.join(OBJ_DIR, os.path.splitext(src)[0] + ".o")
        objs.append(obj)
        path = os.path.join(CSRC, src)
        if force or _stale(obj, [path] + headers):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-x", "cu", "-c", path, "-o", obj]
            jobs.append(cmd)

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("%s failed: %s\n%s\n%s" % (cmd[0], " ".join(cmd), res.stdout, res.stderr))
        if verbose:
            sys.stderr.write(res.stderr)

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as pool:
        list(pool.map(run, jobs))
    if jobs or force or _stale(LIB_PATH, objs):
        run([nvcc, "-shared", "-o", LIB_PATH] + objs + ["-Xlinker", "--no-undefined", "-ldl", "-lpthread"])
    if force or _calls_stale([CALLS_SOURCE] + headers):
        run(_calls_command())
        with open(CALLS_STAMP, "w") as f:
            f.write(_calls_target())
    return LIB_PATH


def _calls_target() -> str:
    """The interpreter and the torch that a binding built now is for: it loads with no others."""
    return "Python %s, torch %s" % (sys.version, importlib.metadata.version("torch"))


def _calls_stale(deps) -> bool:
    if _stale(CALLS_PATH, deps) or not os.path.exists(CALLS_STAMP):
        return True
    with open(CALLS_STAMP) as f:
        return f.read() != _calls_target()


def _calls_command():
    """The binding for torch tensors: an extension module beside the library, which it finds there ($ORIGIN)."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"))
    includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"], os.path.join(ROOT, "include")]
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
             "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI]
            + ["-I" + d for d in includes] + [CALLS_SOURCE, "-o", CALLS_PATH, "-L" + os.path.join(root, "lib"), "-L" + HERE,
                                              "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-l:libdifb200.so",
                                              "-Wl,-rpath,$ORIGIN"])


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
