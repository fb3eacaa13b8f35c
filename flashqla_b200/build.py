"""Build the native code in-tree: ``libfqla_sm100.so`` (the C-ABI library of the CUDA kernels,
nvcc) and ``_host.so`` (the operator's host path against PyTorch's C++ API, g++).

    python -m flashqla_b200.build            # incremental
    python -m flashqla_b200.build --force    # rebuild everything

Only sm_100a code is generated.  Objects go to ``flashqla_b200/csrc/_obj`` and the shared
library next to this file, so that a copy of the source tree carries the built library with it.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(HERE, "libfqla_sm100.so")
HOST_SRC = os.path.join(CSRC, "host")
HOST_LIB = os.path.join(HERE, "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--use_fast_math",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA kernels cannot be built")


def _sources() -> list[str]:
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime() -> float:
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hdrs.append(os.path.join(os.path.dirname(HERE), "include", "fqla.h"))
    return max(os.path.getmtime(h) for h in hdrs)


def _compile(src: str, force: bool, hdr_mtime: float) -> tuple[str, str]:
    obj = os.path.join(OBJ, src[:-3] + ".o")
    path = os.path.join(CSRC, src)
    if (
        not force
        and os.path.exists(obj)
        and os.path.getmtime(obj) > max(os.path.getmtime(path), hdr_mtime)
    ):
        return obj, ""
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", path, "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
    return obj, res.stderr


def _compile_host(src: str, force: bool) -> str:
    """One host source against the headers of the PyTorch that is installed."""
    import torch

    root = os.path.join(os.path.dirname(torch.__file__), "include")
    hdrs = [os.path.join(HOST_SRC, f) for f in os.listdir(HOST_SRC) if f.endswith(".h")]
    hdrs.append(os.path.join(os.path.dirname(HERE), "include", "fqla.h"))
    path, obj = os.path.join(HOST_SRC, src), os.path.join(OBJ, "host_" + src[:-4] + ".o")
    newest = max(os.path.getmtime(f) for f in [path, *hdrs])
    if not force and os.path.exists(obj) and os.path.getmtime(obj) > newest:
        return obj
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-isystem", root, "-isystem", os.path.join(root, "torch", "csrc", "api", "include"),
           "-isystem", os.path.join(cuda, "include"),
           "-isystem", sysconfig.get_paths()["include"], "-c", path, "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {src}:\n{res.stdout}\n{res.stderr}")
    return obj


def _link_host(objs: list[str], force: bool) -> None:
    import torch

    newest = max(os.path.getmtime(f) for f in objs)
    if not force and os.path.exists(HOST_LIB) and os.path.getmtime(HOST_LIB) > newest:
        return
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-shared", "-o", HOST_LIB, *objs, "-L" + libs, "-L" + HERE,
           "-l:libfqla_sm100.so", "-ltorch_python", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda",
           "-lc10", "-Wl,-rpath,$ORIGIN"]
    # the CUDA runtime PyTorch itself loads
    import glob
    rt = [f for d in (libs, os.path.join(os.path.dirname(os.path.dirname(torch.__file__)), "nvidia",
                                         "cuda_runtime", "lib"),
                      os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "lib64"))
          for f in sorted(glob.glob(os.path.join(d, "libcudart*.so.12*")))]
    if rt:
        cmd.append(rt[0])
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link of {HOST_LIB} failed:\n{res.stdout}\n{res.stderr}")


def build_library(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    hdr_mtime = _deps_mtime()
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        host = [pool.submit(_compile_host, f, force) for f in sorted(os.listdir(HOST_SRC))
                if f.endswith(".cpp")]
        results = list(pool.map(lambda s: _compile(s, force, hdr_mtime), _sources()))
        host_objs = [f.result() for f in host]
    objs = [o for o, _ in results]
    logs = "".join(log for _, log in results)
    if logs:
        with open(os.path.join(OBJ, "ptxas.log"), "a") as f:
            f.write(logs)
    if verbose and logs:
        print(logs, file=sys.stderr)
    if force or not os.path.exists(LIB) or any(
        os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs
    ):
        cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-lcudart"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _link_host(host_objs, force)
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
