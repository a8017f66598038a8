"""Builds the C-ABI shared library ``libnb_attn.so`` with nvcc for sm_100a and the PyTorch binding
``_nb_torch.so`` (the custom ops' native bodies, linked to the former) next to this package.

Both are compiled in-tree (not into a JIT cache) so that the built files sit beside the sources they
came from. ``python -m nanobrain_b200.build`` rebuilds them.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libnb_attn.so"
SOURCES = [CSRC / "nb_attn.cu", CSRC / "encoder.cu"]
HEADERS = sorted(CSRC.glob("*.cuh")) + sorted((PKG_DIR.parent / "include").glob("nb_*.h"))

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "-shared",
    "-Xcompiler",
    "-fPIC",
]


TORCH_LIB_PATH = PKG_DIR / "_nb_torch.so"
TORCH_SOURCES = [CSRC / "torch_ops.cpp", CSRC / "torch_encoder.cpp"]
TORCH_HEADERS = [CSRC / "torch_common.h"] + sorted((PKG_DIR.parent / "include").glob("nb_*.h"))


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; set CUDA_HOME")
    return nvcc


def _stale(lib: Path, sources) -> bool:
    if not lib.exists():
        return True
    built = lib.stat().st_mtime
    return any(src.stat().st_mtime > built for src in sources)


def is_stale() -> bool:
    return _stale(LIB_PATH, SOURCES + HEADERS) or _stale(TORCH_LIB_PATH, TORCH_SOURCES + TORCH_HEADERS)


def _run(cmd, what: str, verbose: bool) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"{what} failed:\n" + proc.stdout + proc.stderr)


def _build_abi(verbose: bool) -> None:
    cmd = [find_nvcc(), *NVCC_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    _run(cmd + ["-o", str(LIB_PATH), *map(str, SOURCES)], "nvcc", verbose)


def _build_torch(verbose: bool) -> None:
    """The binding has no device code: a host compiler, torch's headers and libraries, and a run path
    that finds ``libnb_attn.so`` beside it."""
    import sysconfig

    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(find_nvcc()).resolve().parent.parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include",
                Path(sysconfig.get_paths()["include"])]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-DTORCH_EXTENSION_NAME={TORCH_LIB_PATH.stem}"]
    for inc in includes:
        cmd += ["-isystem", str(inc)]
    cmd += ["-o", str(TORCH_LIB_PATH), *map(str, TORCH_SOURCES), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda",
            "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-L{PKG_DIR}", f"-l:{LIB_PATH.name}",
            "-Wl,-rpath,$ORIGIN"]
    _run(cmd, "the binding's compilation", verbose)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile what is missing or older than its sources; returns the C-ABI library's path."""
    if force or _stale(LIB_PATH, SOURCES + HEADERS):
        _build_abi(verbose)
    if force or _stale(TORCH_LIB_PATH, TORCH_SOURCES + TORCH_HEADERS):
        _build_torch(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose="-v" in sys.argv))
