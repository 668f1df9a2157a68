"""In-tree build of libyskn_kv4.so (nvcc, sm_100a only) and of the Python-side argument marshalling `_host.so` (g++).
`python -m yasakani_b200.build [--force] [-v]`.  Objects are kept under build/, so that a changed source recompiles alone."""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libyskn_kv4.so")
HOST = os.path.join(HERE, "_host.so")
HOST_SRC = os.path.join(CSRC, "host_py.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _headers() -> list[str]:
    return glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))


def _older(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(p) > t for p in deps)


def _stale() -> bool:
    return _older(LIB, sources() + _headers()) or _older(HOST, [HOST_SRC] + _headers())


def _run(cmd: list[str]) -> str:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(cmd[0] + " failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return r.stderr


def _build_host() -> None:
    import torch
    t = os.path.join(os.path.dirname(torch.__file__))
    cuda = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          f"-I{t}/include", f"-I{t}/include/torch/csrc/api/include", f"-I{cuda}/include", "-I" + sysconfig.get_paths()["include"], HOST_SRC, "-o", HOST,
          "-L" + HERE, "-l:libyskn_kv4.so", f"-L{t}/lib", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"])


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into one shared library next to this file, and the extension that calls it."""
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC") or "nvcc"
    os.makedirs(OBJ, exist_ok=True)

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, os.path.basename(src) + ".o")
        if force or _older(obj, [src] + _headers()):
            log = _run([nvcc, *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", "-o", obj, src])
            if verbose:
                sys.stderr.write(log)
        return obj

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        objs = list(pool.map(compile_one, sources()))
    if force or _older(LIB, objs):
        _run([nvcc, *NVCC_FLAGS, "-shared", "-lcuda", "-o", LIB, *objs])
    if force or _older(HOST, [HOST_SRC, LIB]):
        _build_host()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
