"""Build librgd_b200.so in-tree with nvcc for sm_100a.

    python -m rgd_triton_b200.build [--force] [--verbose]

Every ``csrc/*.cu`` is compiled to an object file under ``csrc/build/`` (in
parallel, skipped when the object is newer than the source and the headers) and
linked into ``rgd_triton_b200/librgd_b200.so``; ``csrc/host/torch_host.cpp``, the
native host path on top of the C ABI, becomes the extension module
``rgd_triton_b200/_host.so``.  No GPU is needed to build.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import importlib.metadata
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = CSRC / "build"
LIB = PKG / "librgd_b200.so"
HOST_SRC = CSRC / "host" / "torch_host.cpp"
HOST_LIB = PKG / "_host.so"
HOST_STAMP = OBJ / "host_versions"       # the torch and Python that _host.so was built against
INCLUDE = PKG.parent / "include"

NVCC_FLAGS = [
    "-std=c++17",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put /usr/local/cuda/bin on PATH")


def _deps_mtime() -> float:
    hdrs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(INCLUDE.glob("*.h"))
    return max((h.stat().st_mtime for h in hdrs), default=0.0)


def _compile(src: Path, force: bool, verbose: bool, ptxas_v: bool) -> tuple[Path, str]:
    obj = OBJ / (src.stem + ".o")
    newest_dep = max(src.stat().st_mtime, _deps_mtime(), Path(__file__).stat().st_mtime)
    if not force and obj.exists() and obj.stat().st_mtime >= newest_dep:
        return obj, ""
    cmd = [_nvcc(), *NVCC_FLAGS, f"-I{INCLUDE}", "-c", str(src), "-o", str(obj)]
    if ptxas_v:
        cmd[1:1] = ["-Xptxas", "-v"]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
    return obj, res.stderr


def _build_host(force: bool, verbose: bool) -> None:
    """The extension module (plain C++ against torch's headers; it finds librgd_b200.so at run time)."""
    newest_dep = max(p.stat().st_mtime for p in (HOST_SRC, INCLUDE / "rgd_b200.h", Path(__file__)))
    versions = f"torch {importlib.metadata.version('torch')}, Python {sys.version}"
    if not force and HOST_LIB.exists() and HOST_LIB.stat().st_mtime >= newest_dep and \
            HOST_STAMP.exists() and HOST_STAMP.read_text() == versions:
        return
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    torch_lib = Path(torch.__file__).resolve().parent / "lib"
    cuda_inc = Path(_nvcc()).resolve().parent.parent / "include"
    incs = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], str(cuda_inc)]
    cmd = ["g++", "-std=c++17", "-O2", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{i}" for i in incs], str(HOST_SRC), "-o", str(HOST_LIB), f"-L{torch_lib}",
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-ldl"]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC.name}:\n{res.stdout}\n{res.stderr}")
    HOST_STAMP.write_text(versions)


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def build(force: bool = False, verbose: bool = False, ptxas_v: bool = False) -> Path:
    """Compile and link the library; returns its path."""
    OBJ.mkdir(parents=True, exist_ok=True)
    srcs = sources()
    if not srcs:
        raise RuntimeError(f"no CUDA sources under {CSRC}")
    logs = []
    with cf.ThreadPoolExecutor(max_workers=min(len(srcs) + 1, os.cpu_count() or 4)) as ex:
        host = ex.submit(_build_host, force, verbose)
        futs = [ex.submit(_compile, s, force, verbose, ptxas_v) for s in srcs]
        objs = []
        for f in futs:
            o, log = f.result()
            objs.append(o)
            if log:
                logs.append(log)
        host.result()
    if ptxas_v:
        print("\n".join(logs))
    need_link = force or not LIB.exists() or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs)
    if need_link:
        cmd = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a",
               "-o", str(LIB), *map(str, objs)]
        if verbose:
            print(" ".join(cmd), flush=True)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB


def main(argv=None) -> int:
    ap = argparse.ArgumentParser(description=__doc__)
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--ptxas-v", action="store_true", help="print registers / spills / shared memory per kernel")
    a = ap.parse_args(argv)
    lib = build(a.force, a.verbose, a.ptxas_v)
    print(lib)
    return 0


if __name__ == "__main__":
    sys.exit(main())
