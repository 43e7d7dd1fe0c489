"""Builds libmoba_b200.so in-tree with nvcc for sm_100a, and the autograd node with the host compiler.

    python -m moba_triton_b200.build [--force] [--verbose]

Every csrc/*.cu is compiled to an object (in parallel) and linked into
`moba_triton_b200/libmoba_b200.so`. The library links the static CUDA runtime
only; the driver entry points it needs (tensor-map encoding) are resolved at
run time, so it loads on machines without a GPU driver. csrc/autograd.cpp becomes
`moba_triton_b200/_autograd.so`, a torch extension module without device code.
"""

import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libmoba_b200.so")
AUTOGRAD_SRC = os.path.join(CSRC, "autograd.cpp")
AUTOGRAD = os.path.join(PKG, "_autograd.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _newest_dep() -> float:
    deps = glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(PKG, "..", "include", "*.h"))
    return max(os.path.getmtime(p) for p in deps)


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def build_autograd(force: bool = False) -> str:
    header = os.path.join(PKG, "..", "include", "moba_b200.h")
    if not force and os.path.exists(AUTOGRAD) and os.path.getmtime(AUTOGRAD) >= max(map(os.path.getmtime, (AUTOGRAD_SRC, header))):
        return AUTOGRAD
    import torch
    from torch.utils import cpp_extension
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    includes = [*cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_API_INCLUDE_EXTENSION_H",
           "-DTORCH_EXTENSION_NAME=_autograd", *(f"-isystem{i}" for i in includes), AUTOGRAD_SRC, "-o", AUTOGRAD,
           f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("build of _autograd.so failed")
    return AUTOGRAD


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles what is out of date and returns the library path."""
    build_autograd(force)
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= _newest_dep():
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    newest_header = max([os.path.getmtime(p) for p in glob.glob(os.path.join(CSRC, "*.cuh"))
                         + glob.glob(os.path.join(PKG, "..", "include", "*.h"))] or [0.0])

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if (not force and os.path.exists(obj)
                and os.path.getmtime(obj) >= max(os.path.getmtime(src), newest_header)):
            return obj
        cmd = [_nvcc(), *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", src, "-o", obj]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or res.returncode:
            sys.stderr.write(res.stdout + res.stderr)
        if res.returncode:
            raise RuntimeError(f"nvcc failed on {src}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, sources()))
    # drop objects whose source no longer exists
    keep = set(objs)
    for stale in glob.glob(os.path.join(OBJ, "*.o")):
        if stale not in keep:
            os.remove(stale)
    cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-cudart", "static"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("link of libmoba_b200.so failed")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
