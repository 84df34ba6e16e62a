"""Builds ``libpkda_b200.so`` (the C-ABI library, nvcc for sm_100a) and ``_native.so`` (the
torch host layer on top of it, g++) in-tree.

    python -m delta_feedback_experiment_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  The libraries are rebuilt only when a source
file is newer than an existing ``.so``, when ``_native.so`` was built for another
torch, or with ``--force``.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

from . import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB_PATH, NATIVE_PATH = _lib.LIB_PATH, _lib.NATIVE_PATH
OBJ_DIR = os.path.join(HERE, "build")

SOURCES = ["pkda_abi.cu", "pkda_recurrent.cu", "pkda_chunk_fwd.cu", "pkda_chunk_bwd.cu",
           "pkda_static_scratch.cu", "pkda_intra_fwd_tc.cu", "pkda_intra_bwd_tc.cu", "pkda_out_tc.cu", "pkda_scan_tc.cu", "pkda_scan_fwd.cu", "pkda_scan_bwd.cu", "pkda_scan_bwd_tc.cu",
           "pkda_recurrent_bwd.cu", "pkda_qkv_conv.cu", "pkda_norm_gate.cu", "pkda_decode_step.cu", "pkda_controls.cu"]
NATIVE_SOURCE = "pkda_torch.cpp"
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-ftz=true",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; cannot build libpkda_b200.so")
    return exe


def _deps() -> list[str]:
    out = [os.path.join(INCLUDE, "pkda_b200.h"), os.path.abspath(__file__)]  # the flags live in this file
    for name in os.listdir(CSRC):
        out.append(os.path.join(CSRC, name))
    return out


def needs_build() -> bool:
    if not (os.path.exists(LIB_PATH) and _lib.native_is_current()):
        return True
    stamp = min(os.path.getmtime(LIB_PATH), os.path.getmtime(NATIVE_PATH))
    return any(os.path.getmtime(d) > stamp for d in _deps())


def _compile_native() -> str:
    """Object file of the torch host layer (headers and ABI of the running torch)."""
    import sysconfig
    import torch
    from torch.utils.cpp_extension import include_paths
    obj = os.path.join(OBJ_DIR, NATIVE_SOURCE.replace(".cpp", ".o"))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           f'-DPKDA_NATIVE_MARKER="{_lib.native_marker()[:-1].decode()}"', "-I", INCLUDE]
    for inc in [*include_paths("cuda"), sysconfig.get_paths()["include"]]:
        cmd += ["-isystem", inc]
    res = subprocess.run([*cmd, "-c", os.path.join(CSRC, NATIVE_SOURCE), "-o", obj], capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed on {NATIVE_SOURCE}:\n{res.stdout}\n{res.stderr}")
    return obj


def _link_native(obj: str) -> None:
    from torch.utils.cpp_extension import library_paths
    cmd = ["g++", "-shared", "-o", NATIVE_PATH, obj, LIB_PATH, "-Wl,-rpath,$ORIGIN"]
    for path in library_paths("cuda"):
        cmd += ["-L", path]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB_PATH
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> tuple[str, str]:
        obj = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{res.stdout}\n{res.stderr}")
        return obj, res.stderr

    with ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as pool:
        native = pool.submit(_compile_native)
        results = list(pool.map(compile_one, SOURCES))
    if verbose:
        for _, log in results:
            sys.stderr.write(log)
    native_obj = native.result()
    for path in (LIB_PATH, NATIVE_PATH):  # new files, not new contents: an older build may be loaded right now
        if os.path.exists(path):
            os.unlink(path)
    cmd = [nvcc, "-shared", "-o", LIB_PATH, "-Xlinker", "-soname=libpkda_b200.so", *[o for o, _ in results], "-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _link_native(native_obj)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
