"""Builds ``libtb200.so`` (the C-ABI library of sm_100a kernels) in-tree with nvcc, and ``_native.so`` (the host side of the
operator calls and of the engine, ``csrc/host``) with the C++ compiler against torch and that library.

Run ``python -m taac_2026_b200.build`` after editing anything under ``csrc/``.  nvcc
cross-compiles for sm_100a, so this works on a machine without a GPU.  Object files are
cached under ``csrc/build/`` and rebuilt only when a source or header is newer.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
BUILD = CSRC / "build"
HOST = CSRC / "host"
LIB_PATH = PKG_DIR / "libtb200.so"
NATIVE_PATH = PKG_DIR / "_native.so"
INCLUDE = PKG_DIR.parent / "include"

ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        raise RuntimeError("nvcc not found; the tb200 kernels cannot be built")
    return nvcc


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _headers() -> list[Path]:
    return sorted(CSRC.glob("*.cuh")) + sorted(INCLUDE.glob("*.h"))


def _stale(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def _compile(src: Path, verbose: bool, ptxas_info: bool) -> Path:
    obj = BUILD / (src.stem + ".o")
    if not _stale(obj, [src, *_headers(), Path(__file__)]):
        return obj
    cmd = [_nvcc(), *ARCH_FLAGS, *COMMON_FLAGS, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
    if ptxas_info:
        cmd += ["-Xptxas", "-v"]
    if verbose:
        print(" ".join(cmd), flush=True)
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{proc.stdout}\n{proc.stderr}")
    if ptxas_info:
        print(proc.stderr, flush=True)
    return obj


def _run(cmd: list[str], what: str, verbose: bool) -> None:
    if verbose:
        print(" ".join(cmd), flush=True)
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{proc.stdout}\n{proc.stderr}")


def _host_toolchain() -> Path:
    """A file that names the torch, the interpreter and the compiler that the host module is built with, rewritten (and so newer than
    the objects) when one of them changes: a module built against another torch does not load."""
    import torch

    stamp = BUILD / "host_toolchain.txt"
    text = f"{torch.__version__} {torch.__file__} {sys.version} {os.environ.get('CXX', 'g++')}\n"
    if not stamp.exists() or stamp.read_text() != text:
        stamp.write_text(text)
    return stamp


def _compile_host(src: Path, stamp: Path, verbose: bool) -> Path:
    import torch
    from torch.utils.cpp_extension import include_paths

    obj = BUILD / ("host_" + src.stem + ".o")
    if not _stale(obj, [src, *sorted(HOST.glob("*.h")), *sorted(INCLUDE.glob("*.h")), Path(__file__), stamp]):
        return obj
    cuda_include = Path(_nvcc()).resolve().parent.parent / "include"
    paths = [*include_paths(), sysconfig.get_paths()["include"], str(cuda_include)]
    _run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_native",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *(f"-I{p}" for p in paths), "-c", str(src), "-o", str(obj)],
         f"host compiler for {src.name}", verbose)
    return obj


def _link_host(objs: list[Path], verbose: bool) -> None:
    import torch

    torch_lib = Path(torch.__file__).resolve().parent / "lib"
    # The C++ runtime is torch's shared one, by name: a compiler that has the static library alone would put a second runtime into the
    # module, and a stream or an exception that crosses between the two ends the process.
    _run([os.environ.get("CXX", "g++"), "-shared", "-o", str(NATIVE_PATH), *map(str, objs), f"-L{PKG_DIR}", "-l:libtb200.so", f"-L{torch_lib}",
          "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda", "-lc10", "-l:libstdc++.so.6", "-Wl,-rpath,$ORIGIN"],
         "link of the host module", verbose)


def build(*, verbose: bool = False, force: bool = False, ptxas_info: bool = False) -> Path:
    """Compile every ``csrc/*.cu`` for sm_100a and link ``libtb200.so``, then the host module.  Returns the library's path."""
    BUILD.mkdir(parents=True, exist_ok=True)
    if force:
        for obj in BUILD.glob("*.o"):
            obj.unlink()
    srcs = sources()
    stamp = _host_toolchain()
    with ThreadPoolExecutor(max_workers=min(len(srcs), os.cpu_count() or 1)) as pool:
        host = [pool.submit(_compile_host, s, stamp, verbose) for s in sorted(HOST.glob("*.cpp"))]
        objs = list(pool.map(lambda s: _compile(s, verbose, ptxas_info), srcs))
        host_objs = [h.result() for h in host]
    if force or _stale(LIB_PATH, objs):
        cmd = [_nvcc(), *ARCH_FLAGS, "-shared", "-o", str(LIB_PATH), *map(str, objs), "-lcudart"]
        if verbose:
            print(" ".join(cmd), flush=True)
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode != 0:
            raise RuntimeError(f"link failed:\n{proc.stdout}\n{proc.stderr}")
    if force or _stale(NATIVE_PATH, [*host_objs, LIB_PATH, Path(__file__), stamp]):
        _link_host(host_objs, verbose)
    return LIB_PATH


if __name__ == "__main__":
    path = build(verbose=True, force="--force" in sys.argv, ptxas_info="--ptxas" in sys.argv)
    print(path)
