"""Build ``libhades_b200.so`` (the C-ABI library) in-tree with nvcc for sm_100a.

(and ``_native``, the CPython extension that calls it on the hot paths.)
``python -m hades_b200._build`` or ``hades_b200._build.build()``.  Each ``csrc/*.cu``
is compiled to an object under ``build/`` (skipped when up to date) and linked into
``hades_b200/libhades_b200.so``.  No torch headers are involved there: the library is plain
CUDA behind ``include/hades_b200.h``; ``csrc/py/native.cpp`` is compiled against torch.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
OBJ = ROOT / "build" / "obj"
LIB = PKG / "libhades_b200.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "--extended-lambda",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build hades_b200")
    return exe


def _deps_mtime() -> float:
    hdrs = list(CSRC.glob("*.cuh")) + list((ROOT / "include").glob("*.h"))
    return max(p.stat().st_mtime for p in hdrs)


def _compile(src: Path, force: bool) -> tuple[Path, str]:
    obj = OBJ / (src.stem + ".o")
    if not force and obj.exists() and obj.stat().st_mtime >= max(src.stat().st_mtime, _deps_mtime()):
        return obj, ""
    cmd = [_nvcc(), *NVCC_FLAGS, "-I", str(ROOT / "include"), "-c", str(src), "-o", str(obj)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
    obj.with_suffix(".ptxas").write_text(r.stderr)  # registers and spills of every kernel
    return obj, r.stderr


def native_path() -> Path:
    return PKG / ("_native" + sysconfig.get_config_var("EXT_SUFFIX"))


def _build_native(force: bool) -> None:
    """The extension links against libhades_b200.so beside it (the one that ctypes loads too)."""
    src, out = CSRC / "py" / "native.cpp", native_path()
    header = ROOT / "include" / "hades_b200.h"
    if not force and out.exists() and out.stat().st_mtime >= max(src.stat().st_mtime, header.stat().st_mtime):
        return
    import torch

    tdir = Path(torch.__file__).parent
    cuda = Path(_nvcc()).resolve().parent.parent
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else (shutil.which("g++") or "g++")
    cmd = [gxx, "-O2", "-std=c++17", "-fPIC", "-shared", str(src), "-o", str(out),
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", str(ROOT / "include"), "-I", str(tdir / "include"), "-I", str(tdir / "include/torch/csrc/api/include"),
           "-I", sysconfig.get_paths()["include"], "-I", str(cuda / "include"),
           "-L", str(PKG), "-lhades_b200", "-L", str(tdir / "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu",
           "-ltorch_cuda", "-lc10", "-lc10_cuda", "-L", str(cuda / "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{gxx} failed for {src.name}:\n{r.stdout}\n{r.stderr}")


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every CUDA source for sm_100a and link the shared library."""
    OBJ.mkdir(parents=True, exist_ok=True)
    srcs = sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        results = list(ex.map(lambda s: _compile(s, force), srcs))
    objs = [o for o, _ in results]
    if verbose:
        for _, log in results:
            if log:
                sys.stderr.write(log)
    newest = max(o.stat().st_mtime for o in objs)
    if force or not LIB.exists() or LIB.stat().st_mtime < newest:
        cmd = [_nvcc(), "-shared", "-o", str(LIB), *map(str, objs),
               "-gencode", "arch=compute_100a,code=sm_100a",
               "-Xcompiler", "-fPIC", "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_native(force)
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
