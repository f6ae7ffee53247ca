"""Build the C-ABI shared library ``rfa_b200/csrc/librfa_b200.so`` with nvcc for sm_100a, and ``rfa_b200/_native.so``, the
tensor-level calls over it (``csrc/torch_ops.cpp``, against this interpreter's torch).

    python -m rfa_b200.build [--force] [--verbose]

Each ``csrc/*.cu`` is compiled to an object file (in parallel) and linked into
one shared library that exports the ``extern "C"`` entry points declared in
``include/rfa_b200.h``.  nvcc cross-compiles, so no GPU is needed to build.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(CSRC, "librfa_b200.so")
NATIVE_SRC, NATIVE = os.path.join(CSRC, "torch_ops.cpp"), os.path.join(HERE, "_native.so")
NATIVE_KEY = os.path.join(HERE, "_native.key")      # what the module was built for (see native_key)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--extended-lambda", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the rfa_b200 library can only be built with the CUDA toolkit")
    return exe


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(os.path.dirname(HERE), "include", "rfa_b200.h"))
    return hs


def stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def compile_one(src: str, verbose: bool) -> str:
    obj = src[:-3] + ".o"
    if stale(obj, [src] + headers()):
        cmd = [nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        log = r.stdout + r.stderr
        with open(obj + ".log", "w") as f:
            f.write(" ".join(cmd) + "\n" + log)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {os.path.basename(src)}:\n{log}")
        if verbose:
            print(log)
    return obj


def native_key() -> str:
    """The interpreter and the torch an extension module is tied to."""
    import torch
    return f"torch {torch.__version__} cxx11-abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} python {sys.implementation.cache_tag}\n"


def native_stale() -> bool:
    if stale(NATIVE, [NATIVE_SRC, os.path.join(os.path.dirname(HERE), "include", "rfa_b200.h")]) or not os.path.exists(NATIVE_KEY):
        return True
    with open(NATIVE_KEY) as f:
        return f.read() != native_key()


def build_native() -> str:
    """The torch extension module: links the C-ABI library beside it (found through its own path)."""
    if native_stale():
        import sysconfig

        import torch
        from torch.utils.cpp_extension import include_paths
        root = os.path.dirname(torch.__file__)
        cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc())))
        incs = [*include_paths(), sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               *[f"-I{i}" for i in incs], NATIVE_SRC, "-o", NATIVE, "-L" + CSRC, "-l:librfa_b200.so", "-L" + os.path.join(root, "lib"),
               "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN/csrc"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("building _native.so failed:\n" + r.stdout + r.stderr)
        with open(NATIVE_KEY, "w") as f:
            f.write(native_key())
    return NATIVE


def build(force: bool = False, verbose: bool = False) -> str:
    srcs = sources()
    if force:
        for s in srcs:
            if os.path.exists(s[:-3] + ".o"):
                os.remove(s[:-3] + ".o")
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: compile_one(s, verbose), srcs))
    if stale(LIB, objs):
        cmd = [nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    if force and os.path.exists(NATIVE):
        os.remove(NATIVE)
    build_native()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
