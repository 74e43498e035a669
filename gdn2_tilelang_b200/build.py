"""Build ``libgdn2_b200.so`` in-tree with nvcc for sm_100a (cross-compiles without a GPU), and beside it the host
extension ``_gdn2_host.*.so`` (g++, PyTorch's headers) that makes the short calls without going through Python. The package
works without the extension: a failure to build it is a warning.

    python -m gdn2_tilelang_b200.build [--force] [--verbose]
"""

from __future__ import annotations

import argparse
import concurrent.futures
import os
import pathlib
import shutil
import subprocess
import sys
import warnings

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libgdn2_b200.so"
HOST_SRC = CSRC / "host" / "binding.cpp"


def host_lib() -> pathlib.Path:
    """The host extension for THIS Python and PyTorch: it is linked against PyTorch's C++ interface, so one that was built
    under another version must not be loaded."""
    import re
    import sysconfig

    import torch

    tag = re.sub(r"[^A-Za-z0-9_]+", "_", f"torch_{torch.__version__}_{sysconfig.get_config_var('SOABI')}")
    return PKG / f"_gdn2_host.{tag}.so"


NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall",
]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the CUDA kernels cannot be built")
    return nvcc


def _stale(target: pathlib.Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    nvcc = find_nvcc()
    OBJ.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "gdn2_b200.h"]
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: pathlib.Path):
        obj = OBJ / (src.stem + ".o")
        if force or _stale(obj, [src, *headers]):
            cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(src), "-o", str(obj)]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src.name}:\n{r.stdout}\n{r.stderr}")
            if verbose:
                sys.stderr.write(r.stderr)
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        objs = list(ex.map(compile_one, sources))
    if force or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    try:
        build_host(force)
    except (RuntimeError, OSError) as e:
        warnings.warn(f"the host extension was not built, short calls go through Python: {e}")
    return LIB


def build_host_if_missing() -> pathlib.Path:
    target = host_lib()
    return target if target.exists() else build_host()


def build_host(force: bool = False) -> pathlib.Path:
    header = PKG.parent / "include" / "gdn2_b200.h"
    target = host_lib()
    if force or _stale(target, [HOST_SRC, header]):
        import sysconfig

        import torch
        from torch.utils.cpp_extension import include_paths

        cuda = pathlib.Path(find_nvcc()).resolve().parent.parent
        includes = [*include_paths(), sysconfig.get_paths()["include"], str(cuda / "include")]
        torch_lib = pathlib.Path(torch.__file__).parent / "lib"
        tmp = target.with_suffix(f".{os.getpid()}.tmp")
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
               *(f"-I{i}" for i in includes), str(HOST_SRC), "-o", str(tmp), f"-L{torch_lib}", "-lc10", "-lc10_cuda",
               "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-ltorch", f"-L{PKG}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"g++ failed on {HOST_SRC.name}:\n{r.stdout}\n{r.stderr}")
        os.replace(tmp, target)
    return target


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
