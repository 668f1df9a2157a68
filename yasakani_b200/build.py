"""In-tree build of libyskn_kv4.so (nvcc, sm_100a only) and of the Python-side argument marshalling `_host-<id>.so` (g++, needs torch).
`python -m yasakani_b200.build [--force] [-v]`.  Objects are kept under build/, so that a changed source recompiles alone."""
from __future__ import annotations

import glob
import hashlib
import importlib.util
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libyskn_kv4.so")
STAMP = os.path.join(OBJ, "lib.stamp")              # flags and sources of the library that stands
HOST_SRC = os.path.join(CSRC, "host_py.cpp")
ABI = os.path.join(HERE, "..", "include", "yskn_kv4_abi.h")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _headers() -> list[str]:
    return glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))


def _older(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(p) > t for p in deps)


def _recipe() -> str:
    return "\n".join(NVCC_FLAGS + [os.path.basename(p) for p in sources()])


def _same_recipe() -> bool:
    try:
        with open(STAMP) as f:
            return f.read() == _recipe()
    except OSError:
        return False


def _stale() -> bool:
    return _older(LIB, sources() + _headers()) or not _same_recipe()


def _run(cmd: list[str]) -> str:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(cmd[0] + " failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return r.stderr


def _into(target: str, cmd: list[str]) -> None:
    """Run `cmd` with its output in the place of "{out}", then move it over `target`: a process that has the old file loaded keeps it whole."""
    tmp = f"{target}.{os.getpid()}.tmp"
    try:
        _run([tmp if c == "{out}" else c for c in cmd])
        os.replace(tmp, target)
    finally:
        if os.path.exists(tmp):
            os.remove(tmp)


def host_path() -> str:
    """Where the extension for this torch, this Python, this source and this ABI header belongs: one that was built for others has another name."""
    import torch
    h = hashlib.sha1()
    for p in (HOST_SRC, ABI):
        with open(p, "rb") as f:
            h.update(f.read())
    h.update(repr((torch.__version__, int(torch._C._GLIBCXX_USE_CXX11_ABI), sysconfig.get_config_var("SOABI"), HOST_FLAGS)).encode())
    return os.path.join(HERE, f"_host-{h.hexdigest()[:12]}.so")


def build_host(force: bool = False) -> str:
    """Compile the extension against the library that stands (which is not touched)."""
    import torch
    path = host_path()
    if force or not os.path.exists(path):
        t = os.path.dirname(torch.__file__)
        cuda = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
        _into(path, ["g++", *HOST_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                     f"-I{t}/include", f"-I{t}/include/torch/csrc/api/include", f"-I{cuda}/include", "-I" + sysconfig.get_paths()["include"], HOST_SRC,
                     "-o", "{out}", "-L" + HERE, "-l:libyskn_kv4.so", f"-L{t}/lib", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
                     "-Wl,-rpath,$ORIGIN"])
        for old in glob.glob(os.path.join(HERE, "_host*.so")):
            if old != path:
                os.remove(old)
    return path


def build_lib(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into one shared library next to this file (needs nvcc only)."""
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC") or "nvcc"
    os.makedirs(OBJ, exist_ok=True)
    all_of_it = force or not _same_recipe()

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, os.path.basename(src) + ".o")
        if all_of_it or _older(obj, [src] + _headers()):
            log = _run([nvcc, *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", "-o", obj, src])
            if verbose:
                sys.stderr.write(log)
        return obj

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        objs = list(pool.map(compile_one, sources()))
    _into(LIB, [nvcc, *NVCC_FLAGS, "-shared", "-lcuda", "-o", "{out}", *objs])
    with open(STAMP, "w") as f:
        f.write(_recipe())
    return LIB


def build(force: bool = False, verbose: bool = False) -> str:
    """The library, and the extension that calls it where there is a torch to build it for (a C caller needs neither torch nor g++)."""
    lib = build_lib(force, verbose)
    if importlib.util.find_spec("torch") is not None:
        build_host(force)
    return lib


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
