"""Build recipe of the native code: every ``csrc/*.cu`` compiled for sm_100a with nvcc into
``libsplinekv_b200.so`` (the C ABI, no torch types), and ``csrc/skv_host.cpp`` (the operators' host path on
top of it, against torch's headers) into ``_host.so``, both next to this file (in-tree, so that the built
files travel with the source tree).  ``python -m sparsespline_ffn_b200.build`` rebuilds them."""
from __future__ import annotations

import concurrent.futures
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_PATH = os.path.join(HERE, "libsplinekv_b200.so")
HOST_PATH = os.path.join(HERE, "_host.so")
OBJ_DIR = os.path.join(CSRC, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _headers() -> list[str]:
    return glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(os.path.dirname(HERE), "include", "*.h"))


def _newer(target: str, deps: list[str]) -> bool:
    return os.path.exists(target) and all(os.path.getmtime(d) <= os.path.getmtime(target) for d in deps)


def is_fresh() -> bool:
    return _newer(LIB_PATH, sources() + _headers()) and _newer(HOST_PATH, [os.path.join(CSRC, "skv_host.cpp"), *_headers()])


def _run(cmd: list[str], verbose: bool = False) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError("build step failed:\n" + " ".join(cmd) + "\n" + proc.stdout + proc.stderr)


def _host_command() -> list[str]:
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}/include",
            f"-I{sysconfig.get_paths()['include']}", os.path.join(CSRC, "skv_host.cpp"), "-o", HOST_PATH,
            f"-L{HERE}", "-lsplinekv_b200", f"-L{root}/lib", "-ltorch_python", "-ltorch_cpu", "-ltorch", "-lc10", "-lc10_cuda",
            "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is older than its sources (everything with ``force``)."""
    if not force and is_fresh():
        return LIB_PATH
    nvcc = os.environ.get("NVCC", "nvcc")
    os.makedirs(OBJ_DIR, exist_ok=True)
    jobs = []
    objects = []
    for src in sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objects.append(obj)
        if force or not _newer(obj, [src, *_headers()]):
            jobs.append([nvcc, *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", src, "-o", obj])
    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, min(6, (os.cpu_count() or 2) - 2))) as pool:
        list(pool.map(lambda cmd: _run(cmd, verbose), jobs))
    _run([nvcc, *NVCC_FLAGS, "-shared", "-Xlinker", "-soname=" + os.path.basename(LIB_PATH), *objects, "-o", LIB_PATH])
    _run(_host_command(), verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--fast" not in sys.argv, verbose="-v" in sys.argv))
