"""In-tree build of libtuna_b200.so (nvcc, sm_100a only).

The shared library is the product's only native artefact: hand-written CUDA
kernels behind a C ABI (include/tuna_b200.h).  It is built next to the sources
so that it travels with the tree; nothing is JIT-compiled at import time.
"""

from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

from . import _lib

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
LIB = HERE / "libtuna_b200.so"
FAST_CALL = HERE / ("_fast_call" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = ["tuna_api.cu", "host_util.cu", "dequant_sm100a.cu", "quantize_sm100a.cu", "gemm_stream_sm100a.cu", "gemm_tstream_sm100a.cu", "gemm_pair_sm100a.cu", "exchange_sm100a.cu", "ref_symbols.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(d).stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every kernel source for sm_100a and link the shared library."""
    from . import make_configs

    make_configs.generate()
    headers = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(CSRC.glob("*.inc")) + [
        HERE.parent / "include" / "tuna_b200.h"
    ]
    objdir = HERE / "build"
    objdir.mkdir(exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str):
        obj = objdir / (src + ".o")
        if force or _stale(obj, [CSRC / src] + headers):
            extra = os.environ.get("TUNA_EXTRA_NVCC_FLAGS", "").split()
            cmd = [nvcc] + NVCC_FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + ["-c", str(CSRC / src), "-o", str(obj)]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if verbose or r.returncode:
                sys.stderr.write(r.stdout + r.stderr)
            if r.returncode:
                raise RuntimeError(f"nvcc failed on {src}")
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    if force or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB)] + [str(o) for o in objs]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    _build_fast_call(force)
    return LIB


def _fast_call_stale() -> bool:
    """Whether the extension is older than its sources or was built for another torch or Python than these."""
    return (_stale(FAST_CALL, [CSRC / "fast_call.cpp", HERE.parent / "include" / "tuna_b200.h"])
            or _lib.fast_call_stamp().encode() + b"\0" not in FAST_CALL.read_bytes())


def _build_fast_call(force: bool) -> None:
    """The native front of `ops.matmul` (csrc/fast_call.cpp): an extension module against the headers of the torch it runs with.

    Beside a torch without CUDA there is nothing to build it against, and nothing that would call it."""
    import torch

    root = Path(torch.__file__).resolve().parent
    if not (root / "lib" / "libc10_cuda.so").exists() or not (force or _fast_call_stale()):
        return
    cuda = Path(_nvcc()).resolve().parent.parent if os.path.sep in _nvcc() else Path("/usr/local/cuda")
    include = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include", sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DFAST_CALL_STAMP="{_lib.fast_call_stamp()}"', *(f"-I{p}" for p in include), str(CSRC / "fast_call.cpp"), "-o", str(FAST_CALL),
           f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:  # no Python headers, say: the library is complete without it
        FAST_CALL.unlink(missing_ok=True)
        sys.stderr.write(r.stdout + r.stderr + "fast_call.cpp was not built: matmul will check its calls in Python\n")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
