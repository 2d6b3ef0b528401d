"""In-tree build of libua_b200.so (sm_100a only) with nvcc, and of the extension module _ua_torch.so above it.

    python -m universal_attention_triton_b200.build [--verbose]

The shared library is written next to this file so that it travels with the
source tree; there is no JIT cache and no pip install step.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libua_b200.so")
SOURCES = ["ua_bwd.cu", "ua_fwd.cu", "ua_tiled.cu", "ua_api.cu"]      # compiled side by side
# the tensor plumbing above the library: an extension module, host code only
TORCH_SOURCE = "ua_torch.cpp"
TORCH_PATH = os.path.join(PKG_DIR, "_ua_torch.so")
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return exe


def _run(cmd):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("failed: " + " ".join(cmd[:1] + cmd[-4:]))
    return res


def _stale() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(TORCH_PATH):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(TORCH_PATH))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(os.path.dirname(PKG_DIR), "include", "ua_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library if it is missing or older than its sources; returns its path."""
    if not force and not _stale():
        return LIB_PATH
    with tempfile.TemporaryDirectory() as tmp, ThreadPoolExecutor() as pool:
        objs = [os.path.join(tmp, src + ".o") for src in SOURCES]
        extra = ["-Xptxas", "-v"] if verbose else []
        for res in pool.map(lambda so: _run([_nvcc()] + NVCC_FLAGS + extra + ["-c", os.path.join(CSRC, so[0]), "-o", so[1]]), zip(SOURCES, objs)):
            if verbose:
                sys.stderr.write(res.stdout + res.stderr)
        _run([_nvcc()] + NVCC_FLAGS + ["-shared"] + objs + ["-o", LIB_PATH, "-lcuda"])
    _build_torch_module()
    return LIB_PATH


def _build_torch_module() -> None:
    """The extension module that holds the tensor plumbing; links the library by its place beside it."""
    import sysconfig
    import torch
    from torch.utils.cpp_extension import include_paths
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda_inc = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for inc in include_paths() + [cuda_inc, sysconfig.get_paths()["include"]]:
        cmd += ["-isystem", inc]
    cmd += [os.path.join(CSRC, TORCH_SOURCE), "-o", TORCH_PATH, "-L" + PKG_DIR, "-l:" + os.path.basename(LIB_PATH), "-L" + torch_lib,
            "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    _run(cmd)


if __name__ == "__main__":
    print(build(force=True, verbose="--verbose" in sys.argv))
