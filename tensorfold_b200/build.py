"""Builds ``libtensorfold_b200.so`` in-tree with nvcc for sm_100a (cross-compiles without a GPU), and beside it
``_native.so``, the host path as a CPython extension over torch's C++ tensors (``csrc/native.cpp``, the C++ compiler alone).

    python -m tensorfold_b200.build [--force]

One object per translation unit, compiled in parallel; the matmul template is instantiated once per bit width
(``qmm_inst.cu``, ``qmm_stream_inst.cu`` and ``qmm_window_inst.cu`` with ``-DTF_BITS=b``).
"""

from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from importlib.metadata import version
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OBJ = HERE / "build"
LIB = HERE / "libtensorfold_b200.so"
NATIVE = HERE / "_native.so"
NATIVE_FOR = OBJ / "native.for"       # what _native.so was compiled against
BITS = (2, 3, 4, 5, 6, 8)
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "--threads", "2"]


def _units() -> list[tuple[Path, Path, list[str]]]:
    units = [(CSRC / "qmm_inst.cu", OBJ / f"qmm_b{b}.o", [f"-DTF_BITS={b}"]) for b in BITS]
    units += [(CSRC / "qmm_stream_inst.cu", OBJ / f"qmm_stream_b{b}.o", [f"-DTF_BITS={b}"]) for b in BITS]
    units += [(CSRC / "qmm_window_inst.cu", OBJ / f"qmm_window_b{b}.o", [f"-DTF_BITS={b}"]) for b in BITS if b != 8]
    for src in sorted(CSRC.glob("*.cu")):
        if src.name not in ("qmm_inst.cu", "qmm_stream_inst.cu", "qmm_window_inst.cu"):
            units.append((src, OBJ / (src.stem + ".o"), []))
    return units


def _newest_header() -> float:
    heads = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + [HERE.parent / "include" / "tensorfold_b200.h"]
    return max(h.stat().st_mtime for h in heads)


def _compile(unit) -> str:
    src, obj, defs = unit
    cmd = ["nvcc", *NVCC_FLAGS, *defs, "-c", str(src), "-o", str(obj)]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode:
        raise RuntimeError(f"nvcc failed for {src.name} {defs}:\n{done.stdout}\n{done.stderr}")
    return obj.name


def _native_for() -> str:
    return f"torch {version('torch')}, {sys.implementation.cache_tag}"


def _native_stale() -> bool:
    """Sources or headers are newer, or torch or the interpreter is another one (their C++ interfaces have no stable ABI)."""

    sources = CSRC / "native.cpp", HERE.parent / "include" / "tensorfold_b200.h"
    return (not NATIVE.exists() or NATIVE.stat().st_mtime < max(s.stat().st_mtime for s in sources)
            or not NATIVE_FOR.exists() or NATIVE_FOR.read_text() != _native_for())


def _native() -> str:
    """Compiles the extension module against the torch that will load it."""

    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    heads = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include",
             Path(sysconfig.get_paths()["include"])]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *(f"-I{h}" for h in heads), str(CSRC / "native.cpp"), "-o", str(NATIVE), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda",
           "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-ldl"]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode:
        raise RuntimeError(f"g++ failed for native.cpp:\n{done.stdout}\n{done.stderr}")
    NATIVE_FOR.write_text(_native_for())
    return NATIVE.name


def build(force: bool = False, verbose: bool = False) -> Path:
    OBJ.mkdir(exist_ok=True)
    heads = _newest_header()
    stale = [u for u in _units()
             if force or not u[1].exists() or u[1].stat().st_mtime < max(u[0].stat().st_mtime, heads)]
    jobs = ([_native] if force or _native_stale() else []) + [lambda u=u: _compile(u) for u in stale]
    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as pool:
            for name in pool.map(lambda job: job(), jobs):
                if verbose:
                    print("compiled", name)
    objs = [str(u[1]) for u in _units()]
    if stale or not LIB.exists():
        cmd = ["nvcc", "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(LIB), *objs]
        done = subprocess.run(cmd, capture_output=True, text=True)
        if done.returncode:
            raise RuntimeError(f"link failed:\n{done.stdout}\n{done.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
