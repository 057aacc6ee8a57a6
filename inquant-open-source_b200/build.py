"""Builds libinquant_b200.so and inquant/_host.so in-tree with nvcc for sm_100a (cross-compiles without a GPU)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libinquant_b200.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]
# Per-file flags: the codec must not contract a*b+c into an FMA (bit-exact bytes).
SOURCES = {
    "lib.cu": [],
    "codec.cu": ["-fmad=false"],
    "decode.cu": [],
    "append.cu": [],
    "prefill.cu": [],
    "decode_generic.cu": [],
    "exchange.cu": [],
    "pages.cu": [],
}


HOST = os.path.join(HERE, "inquant", "_host.so")   # CPython extension: host side of the per-layer calls


def build_host(force: bool = False) -> str:
    """Builds inquant/_host.so against the installed PyTorch, anew for another PyTorch or Python."""
    import sysconfig
    if HERE not in sys.path:
        sys.path.insert(0, HERE)
    import torch
    from inquant._native import host_built_for
    src, stamp, built_for = os.path.join(CSRC, "host.cpp"), os.path.join(HERE, "build", "host.stamp"), host_built_for()
    try:
        with open(stamp) as file:
            force = force or file.read() != built_for
    except OSError:
        force = True
    if force or _stale(HOST, [src, __file__, os.path.join(os.path.dirname(HERE), "include", "inquant_b200.h")]):
        root = os.path.dirname(torch.__file__)
        cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc")))
        includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                    sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
        subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC",
                        f'-DINQ_BUILT_FOR="{built_for}"', f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{i}" for i in includes), src, "-o", HOST,
                        f"-L{os.path.join(root, 'lib')}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"], check=True)
        with open(stamp, "w") as file:
            file.write(built_for)
    return HOST


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    mtime = os.path.getmtime(target)
    return any(os.path.getmtime(d) > mtime for d in deps)


def build_library(force: bool = False, verbose: bool = False) -> str:
    nvcc = os.environ.get("NVCC", "nvcc")
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "inquant_b200.h"))
    objects = []
    build_dir = os.path.join(HERE, "build")
    os.makedirs(build_dir, exist_ok=True)
    running = []
    for name, extra in SOURCES.items():
        src = os.path.join(CSRC, name)
        obj = os.path.join(build_dir, name.replace(".cu", ".o"))
        if force or _stale(obj, [src, __file__] + headers):
            cmd = [nvcc, *ARCH, *COMMON, *extra, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            # the translation units are independent: all stale ones compile at the same time (the
            # decode kernels alone take minutes), which bounds a build from scratch by the longest file
            running.append((cmd, subprocess.Popen(cmd)))
        objects.append(obj)
    failed = [cmd for cmd, process in running if process.wait() != 0]
    if failed:
        raise subprocess.CalledProcessError(1, failed[0])
    if force or _stale(LIB, objects):
        subprocess.run([nvcc, *ARCH, "-shared", "-o", LIB, *objects, "-cudart", "static"], check=True)
    build_host(force)
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
