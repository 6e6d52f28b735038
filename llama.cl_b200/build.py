"""Build the sm_100a shared library ``lib/libq4fc_b200.so`` from ``csrc/*.cu``
and the Python front ``lib/_q4fc_front.so`` from ``csrc/front.cpp``.

In-tree build.  The library needs nvcc only (no torch headers: it has a plain C
ABI); each translation unit is compiled to an object in ``build/`` (in
parallel) and linked with the static CUDA runtime.  The front is host code
against the headers of the installed torch (g++, Python's and torch's headers);
it is linked with the library, and built anew when torch is another one.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB_DIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIB_DIR, "libq4fc_b200.so")
FRONT_SRC = os.path.join(CSRC, "front.cpp")
FRONT = os.path.join(LIB_DIR, "_q4fc_front.so")
FRONT_TORCH = os.path.join(OBJ, "front_torch.txt")  # the torch that FRONT was built against

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if c and os.path.exists(c):
            return c
    raise RuntimeError("nvcc not found")


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _torch_build() -> str:
    import torch

    return f"{torch.__version__} {torch.version.git_version} {os.path.dirname(torch.__file__)}"


def front_stale(deps: list[str]) -> bool:
    if _stale(FRONT, deps) or not os.path.exists(FRONT_TORCH):
        return True
    with open(FRONT_TORCH) as f:
        return f.read() != _torch_build()


def front_command() -> list[str]:
    import sysconfig

    import torch

    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(nvcc()))
    inc = [f"-I{os.path.join(tdir, 'include')}", f"-I{os.path.join(tdir, 'include', 'torch', 'csrc', 'api', 'include')}",
           f"-I{os.path.join(cuda, 'include')}", f"-I{sysconfig.get_paths()['include']}"]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *inc, FRONT_SRC, "-o", FRONT,
            f"-L{os.path.join(tdir, 'lib')}", "-ltorch_python", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda", "-lc10",
            f"-L{os.path.join(cuda, 'lib64')}", "-lcudart", f"-L{LIB_DIR}", "-lq4fc_b200", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(LIB_DIR, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + [
        os.path.join(os.path.dirname(PKG), "include", "q4fc_b200.h")]
    extra = ["-Xptxas", "-v"] if verbose else []
    jobs = []
    objs = []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            jobs.append([nvcc(), *NVCC_FLAGS, *extra, "-c", src, "-o", obj])
    with cf.ThreadPoolExecutor(max_workers=max(1, min(8, len(jobs)))) as ex:
        for res in ex.map(lambda c: subprocess.run(c, capture_output=True, text=True), jobs):
            if verbose or res.returncode:
                sys.stderr.write(res.stdout + res.stderr)
            if res.returncode:
                raise RuntimeError("nvcc failed: " + " ".join(res.args))
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-cudart", "static",
               *objs, "-o", LIB]
        subprocess.run(cmd, check=True)
    if force or front_stale([FRONT_SRC, headers[-1]]):
        subprocess.run(front_command(), check=True)
        with open(FRONT_TORCH, "w") as f:
            f.write(_torch_build())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
