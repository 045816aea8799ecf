"""Build the native code in-tree for sm_100a.

    python -m sps_b200.build [--force] [--verbose]

``libspsattn.so`` (nvcc) holds the kernels behind a plain C ABI, ``_native.so`` (the host compiler,
against PyTorch's headers) the host path of the public functions.  ``sps_b200`` refuses to work
without them.  nvcc cross-compiles, so this runs on a machine without a GPU.
"""

from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from typing import Optional

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libspsattn.so")
NATIVE_PATH = os.path.join(PKG_DIR, "_native.so")
NATIVE_STAMP = os.path.join(PKG_DIR, "_native.stamp")     # what _native.so was built against
ABI_HEADER = os.path.join("..", "..", "include", "spsattn.h")
SOURCES = ["spsattn_api.cu"]
HEADERS = ["common.cuh", "mask.cuh", "prefill_sm100.cuh", "prefill_wide_sm100.cuh", "prefill_bwd_sm100.cuh", "prefill_aux.cuh", "decode.cuh", "decode_sm100.cuh",
           "kv_update.cuh", "model_glue.cuh", "rope.cuh", "cache_fill.cuh", "decoder_step.cuh", "decoder_rows.cuh", "decoder_rows_ring.h", "decoder_rows_plan.h", "prompt.cuh", "device_once.h", ABI_HEADER]
NATIVE_SOURCES = ["native.cpp"]
NATIVE_HEADERS = ["native_engine.h"]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _stale(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    deps = [os.path.join(CSRC, f) for f in sources]
    return any(os.path.getmtime(d) > built for d in deps if os.path.exists(d))


def native_interfaces() -> str:
    """The C++ interfaces that the extension depends on besides its sources: an extension built against
    another torch or Python fails to load, or worse."""
    import torch
    return f"torch {torch.__version__}, Python {sys.version_info.major}.{sys.version_info.minor}"


def built_against() -> Optional[str]:
    """``native_interfaces()`` as they were when the extension was built; None when that is not known."""
    try:
        with open(NATIVE_STAMP) as f:
            return f.read()
    except OSError:
        return None


def _library_stale() -> bool:
    return _stale(LIB_PATH, SOURCES + HEADERS)


def _native_stale() -> bool:
    return (_stale(NATIVE_PATH, NATIVE_SOURCES + NATIVE_HEADERS + [ABI_HEADER])
            or built_against() != native_interfaces())


def is_stale() -> bool:
    return _library_stale() or _native_stale()


def _run(cmd, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("the compiler failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stdout + res.stderr)


def _build_library(verbose: bool) -> None:
    cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "-shared", "-Xcompiler", "-fPIC", "--use_fast_math", "-o", LIB_PATH]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    _run(cmd + [os.path.join(CSRC, s) for s in SOURCES], verbose)


def _build_native(verbose: bool) -> None:
    import torch
    from torch.utils import cpp_extension
    cuda_home = os.path.dirname(os.path.dirname(_nvcc())) or "/usr/local/cuda"
    includes = cpp_extension.include_paths() + [os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    # the compiler on PATH (as nvcc uses it): it links the shared libstdc++ that is in the process with
    # torch; one that links its own copy in statically crashed in stream output
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for inc in includes:
        cmd += ["-isystem", inc]
    cmd += [os.path.join(CSRC, s) for s in NATIVE_SOURCES] + ["-o", NATIVE_PATH]
    for lib in [os.path.join(os.path.dirname(torch.__file__), "lib"), os.path.join(cuda_home, "lib64")]:
        cmd += ["-L" + lib]
    # libspsattn.so is found beside the extension; the others are in the process with torch
    cmd += ["-L" + PKG_DIR, "-lspsattn", "-Wl,-rpath,$ORIGIN", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
            "-ltorch", "-ltorch_python", "-lcudart"]
    _run(cmd, verbose)
    with open(NATIVE_STAMP, "w") as f:
        f.write(native_interfaces())


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _library_stale():
        _build_library(verbose)
    if force or _native_stale():
        _build_native(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
