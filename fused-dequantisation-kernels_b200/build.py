"""Builds libfdk_b200.so (sm_100a only) in-tree, next to the `fdk` package.

    python fused-dequantisation-kernels_b200/build.py [--force]

nvcc cross-compiles without a GPU.  Objects go to csrc/build/, the shared
library to fdk/libfdk_b200.so, the host side of eager calls (a Python extension in C++, without device
code; left out where torch or a host compiler is missing) to fdk/_eager.*.so; all are rebuilt only when a source
is newer, the extension also for another torch.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OBJ = CSRC / "build"
LIB = HERE / "fdk" / "libfdk_b200.so"
EAGER = HERE / "fdk" / ("_eager" + sysconfig.get_config_var("EXT_SUFFIX"))
INCLUDE = HERE.parent / "include"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found; libfdk_b200 cannot be built")
    return exe


def _newest_header() -> float:
    headers = list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    return max(h.stat().st_mtime for h in headers)


def _build_eager(force: bool, verbose: bool) -> bool:
    """Whether the extension is there.  The library does without torch, Python's headers and a host compiler, and the
    package without the extension (its eager calls then take longer), so what is missing here is said and no more.
    Torch's inline code is compiled in: another torch, or another command, makes another extension."""
    source, header, stamp = CSRC / "eager_calls.cpp", INCLUDE / "fdk_b200.h", OBJ / "eager.stamp"
    try:
        import torch

        root = Path(torch.__file__).parent
        cuda = Path(_nvcc()).resolve().parents[1]
        include = [root / "include", root / "include/torch/csrc/api/include", cuda / "include", Path(sysconfig.get_paths()["include"])]
        cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f'-DFDK_TORCH_VERSION="{torch.__version__}"',
               *(f"-I{i}" for i in include), str(source), "-o", str(EAGER), f"-L{root / 'lib'}",
               "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
        made_by = "\n".join(cmd)
        if (not force and EAGER.exists() and EAGER.stat().st_mtime >= max(source.stat().st_mtime, header.stat().st_mtime)
                and stamp.exists() and stamp.read_text() == made_by):
            return True
        EAGER.unlink(missing_ok=True)
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        subprocess.run(cmd, check=True)
        stamp.write_text(made_by)
        return True
    except (ImportError, OSError, subprocess.CalledProcessError) as e:
        EAGER.unlink(missing_ok=True)
        print(f"{EAGER.name} not built ({type(e).__name__}: {e}): eager calls go through Python", file=sys.stderr)
        return False


def build(force: bool = False, verbose: bool = False) -> Path:
    sources = sorted(CSRC.glob("*.cu"))
    OBJ.mkdir(exist_ok=True)
    header_time = _newest_header()
    nvcc = _nvcc()

    def compile_one(src: Path) -> tuple[Path, bool]:
        obj = OBJ / (src.stem + ".o")
        stale = force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, header_time)
        if stale:
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
            if verbose:
                print(" ".join(cmd), file=sys.stderr)
            subprocess.run(cmd, check=True)
        return obj, stale

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        eager = pool.submit(_build_eager, force, verbose)
        results = list(pool.map(compile_one, sources))
        eager.result()
    objs = [o for o, _ in results]
    if force or any(s for _, s in results) or not LIB.exists():
        cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", str(LIB), *map(str, objs)]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
