"""Build recipe of the two in-tree libraries: the kernels behind the C ABI (one ``nvcc`` call, sm_100a only) and the native
host side of the module calls (``csrc/host.cpp``, one ``g++`` call against PyTorch's headers, linked to the first)."""

from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_NAME = "libb200_trimul.so"
LIB_PATH = PKG_DIR / LIB_NAME
NATIVE_PATH = PKG_DIR / "_native.so"
NATIVE_TAG_PATH = PKG_DIR / "_native.tag"  # what NATIVE_PATH was built against
HOST_SOURCE = CSRC / "host.cpp"
HEADER = PKG_DIR.parent / "include" / "b200_trimul.h"

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


def _sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.inc")) + [HEADER]


def is_stale() -> bool:
    if not LIB_PATH.exists():
        return True
    built = LIB_PATH.stat().st_mtime
    return any(src.stat().st_mtime > built for src in _sources())


def native_tag() -> str:
    """The interpreter and the PyTorch that ``_native.so`` is bound to: with another one it does not load, or not rightly."""
    import sysconfig

    import torch

    return f"{sysconfig.get_config_var('SOABI')} torch {torch.__version__} cxx11 abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)}\n"


def native_is_stale() -> bool:
    if not NATIVE_PATH.exists() or not NATIVE_TAG_PATH.exists() or NATIVE_TAG_PATH.read_text() != native_tag():
        return True
    built = NATIVE_PATH.stat().st_mtime
    return any(src.stat().st_mtime > built for src in (HOST_SOURCE, HEADER, Path(__file__)))


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build " + LIB_NAME)
    return nvcc


def _run(cmd: list[str]) -> subprocess.CompletedProcess:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n" + proc.stdout + proc.stderr)
    return proc


def build_native(force: bool = False) -> Path:
    """Compile ``csrc/host.cpp`` into ``_native.so`` beside the package (needs the kernels' library to link to)."""
    if not force and not native_is_stale():
        return NATIVE_PATH
    import sysconfig

    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(find_nvcc()).resolve().parent.parent
    tmp = NATIVE_PATH.with_suffix(".so.tmp")
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_native", "-DTORCH_API_INCLUDE_EXTENSION_H",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f"-I{root}/include",
          f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}/include", f"-I{sysconfig.get_paths()['include']}",
          str(HOST_SOURCE), "-o", str(tmp), f"-L{root}/lib", "-ltorch", "-ltorch_cpu", "-ltorch_python", "-ltorch_cuda", "-lc10", "-lc10_cuda",
          f"-L{PKG_DIR}", f"-l:{LIB_NAME}", "-Wl,-rpath,$ORIGIN"])
    os.replace(tmp, NATIVE_PATH)
    NATIVE_TAG_PATH.write_text(native_tag())
    return NATIVE_PATH


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile ``csrc/trimul_abi.cu`` into ``libb200_trimul.so`` beside the package (no GPU needed), then ``_native.so``."""
    if force or is_stale():
        cmd = [find_nvcc(), *NVCC_FLAGS]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        tmp = LIB_PATH.with_suffix(".so.tmp")
        proc = _run(cmd + ["-o", str(tmp), str(CSRC / "trimul_abi.cu")])
        os.replace(tmp, LIB_PATH)
        if verbose:
            print(proc.stderr)
    build_native(force)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
