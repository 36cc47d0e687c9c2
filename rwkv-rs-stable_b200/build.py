"""Builds ``librwkv7_b200.so`` (the C-ABI library) in-tree with nvcc for sm_100a, and
``rwkv7_b200_torch.so`` (its binding to torch tensors, a CPython module) with g++.

Run as ``python build.py`` from this directory or call :func:`build_library` and
:func:`build_binding`.  Objects go to ``build/`` next to this file; the shared objects are written
beside this file so that they are found without installation.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
BUILD = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "librwkv7_b200.so")

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    # The explicit -gencode form: plain -arch=sm_100a also emits a compute_100
    # target for which ptxas rejects tcgen05.
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall",
    "-I", INCLUDE, "-I", CSRC,
]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build librwkv7_b200.so")
    return nvcc


def sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp")))


def _newer(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


# Named variants of the library: the same sources with extra preprocessor flags, built into their own object
# directory and written beside the product library as librwkv7_b200_<variant>.so.
VARIANTS = {
    "checked": ["-DRWKV7_CHECKED", "-DRWKV7_NVTX"],   # device-side index checks + NVTX ranges (tests only)
}


def build_variant(name: str, force: bool = False) -> str:
    return build_library(force=force, extra_flags=VARIANTS[name], variant=name)


def build_library(force: bool = False, verbose: bool = False, extra_flags: list[str] | None = None,
                  variant: str | None = None) -> str:
    BUILD = os.path.join(HERE, "build", variant) if variant else os.path.join(HERE, "build")
    LIB = os.path.join(HERE, f"librwkv7_b200_{variant}.so") if variant else os.path.join(HERE, "librwkv7_b200.so")
    os.makedirs(BUILD, exist_ok=True)
    nvcc = _nvcc()
    # nvcc's host compiler: the environment's CC/CXX may point at a compiler
    # without the usual runtime pieces, so name the system one explicitly.
    host = ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    flags = NVCC_FLAGS + (extra_flags or [])
    jobs = []
    objs = []
    for src in sources():
        obj = os.path.join(BUILD, os.path.basename(src) + ".o")
        objs.append(obj)
        if force or _newer(obj, [src] + headers):
            cmd = [nvcc, *host, *flags, "-x", "cu", "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, res

    with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        for cmd, res in ex.map(run, jobs):
            if verbose or res.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + res.stdout + res.stderr)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed for {cmd[-3]}")
    if force or jobs or _newer(LIB, objs):
        cmd = [nvcc, *host, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-ldl"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link failed")
    return LIB


def build_binding(force: bool = False) -> str:
    """The torch binding; it opens the library when the package does, and links none of it."""
    src = os.path.join(CSRC, "torch", "binding.cpp")
    out = os.path.join(HERE, "rwkv7_b200_torch.so")
    headers = [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    if not force and not _newer(out, [src] + headers):
        return out
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    lib = os.path.join(root, "lib")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    includes = [INCLUDE, os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = [cxx, "-std=c++17", "-O2", "-fPIC", "-shared", "-Wall", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[a for i in includes for a in ("-isystem" if i != INCLUDE else "-I", i)], src, "-o", out,
           "-L", lib, "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", "-ldl"]
    # (the CUDA runtime torch itself has loaded: a second one would not know its streams' device state)
    cudart = _torch_cudart(root)
    cmd += [cudart] if cudart else ["-L", os.path.join(cuda, "lib64"), "-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + res.stdout + res.stderr)
        raise RuntimeError("building the torch binding failed")
    return out


def _torch_cudart(root: str) -> str | None:
    for base in (os.path.join(root, "lib"), os.path.join(os.path.dirname(root), "nvidia", "cuda_runtime", "lib")):
        if os.path.isdir(base):
            for f in sorted(os.listdir(base)):
                if f.startswith("libcudart") and ".so" in f:
                    return os.path.join(base, f)
    return None


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build_binding(force="--force" in sys.argv))
