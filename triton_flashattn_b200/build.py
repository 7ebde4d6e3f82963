"""Builds libfa_sm100.so (kernels and C ABI, nvcc for sm_100a) and _fa_torch.so (the PyTorch
launch path on top of it, host compiler) in-tree.

Run as ``python -m triton_flashattn_b200.build`` (add ``--force`` to rebuild
everything, ``--verbose`` for ptxas register/shared-memory statistics).  Objects
are rebuilt only when a source or header is newer than them.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
BUILD_DIR = os.path.join(PKG_DIR, "build")
LIB_PATH = os.path.join(PKG_DIR, "libfa_sm100.so")
BINDING_SRC = os.path.join(CSRC, "torch_binding.cpp")
BINDING_PATH = os.path.join(PKG_DIR, "_fa_torch.so")
BINDING_STAMP = os.path.join(BUILD_DIR, "_fa_torch.stamp")
INCLUDE_DIR = os.path.join(os.path.dirname(PKG_DIR), "include")

SOURCES = [
    "fa_api.cu",
    "fa_selftest.cu",
    "fa_fwd.cu",
    "fa_decode.cu",
    "fa_small.cu",
    "fa_copy.cu",
    "fa_bwd_pre.cu",
    "fa_bwd_dkdv.cu",
    "fa_bwd_dq.cu",
    "fa_bwd_dkdv256.cu",
    "fa_bwd_static.cu",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libfa_sm100.so cannot be built")
    return exe


def _headers() -> list[str]:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(INCLUDE_DIR, f) for f in os.listdir(INCLUDE_DIR) if f.endswith(".h")]
    return hs


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every translation unit and link the two shared libraries; returns the kernels' path."""
    os.makedirs(BUILD_DIR, exist_ok=True)
    nvcc = _nvcc()
    headers = _headers()
    srcs = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    flags = [
        "-gencode", "arch=compute_100a,code=sm_100a",
        "-std=c++17", "-O3", "-lineinfo",
        "-Xcompiler", "-fPIC",
        "--expt-relaxed-constexpr",
        "-I", INCLUDE_DIR,
    ]
    if verbose:
        flags += ["-Xptxas", "-v"]

    def compile_one(src: str) -> tuple[str, bool, str]:
        obj = os.path.join(BUILD_DIR, src.replace(".cu", ".o"))
        path = os.path.join(CSRC, src)
        if not force and not _stale(obj, [path] + headers):
            return obj, False, ""
        cmd = [nvcc, *flags, "-c", path, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        return obj, True, r.stderr

    with ThreadPoolExecutor(max_workers=min(len(srcs), os.cpu_count() or 4)) as ex:
        results = list(ex.map(compile_one, srcs))
    objs = [o for o, _, _ in results]
    if verbose:
        for _, _, log in results:
            if log:
                print(log)
    if force or any(c for _, c, _ in results) or _stale(LIB_PATH, objs):
        cmd = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
               "-Xcompiler", "-fPIC"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_binding(force)
    return LIB_PATH


def _binding_key() -> str:
    """What the launch path is compiled against, besides its sources."""
    import torch

    return f"torch {torch.__version__} {torch.version.git_version} {sysconfig.get_config_var('SOABI')}\n"


def _binding_stale() -> bool:
    """Older than its sources, or built against another torch or Python than the running one."""
    if _stale(BINDING_PATH, [BINDING_SRC] + [h for h in _headers() if h.endswith(".h")]):
        return True
    try:
        with open(BINDING_STAMP) as f:
            return f.read() != _binding_key()
    except OSError:
        return True


def build_binding(force: bool = False) -> str:
    """Compile the PyTorch launch path against the installed torch and link it to libfa_sm100.so
    (found beside it at run time); returns its path."""
    import torch

    if not force and not _binding_stale():
        return BINDING_PATH
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = [
        shutil.which("g++") or "c++", "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
        "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
        "-I", sysconfig.get_path("include"), "-I", os.path.join(cuda, "include"), "-I", INCLUDE_DIR,
        BINDING_SRC, "-o", BINDING_PATH,
        "-L", PKG_DIR, "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN",
        "-L", os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
    ]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {BINDING_SRC}:\n{r.stdout}\n{r.stderr}")
    with open(BINDING_STAMP, "w") as f:
        f.write(_binding_key())
    return BINDING_PATH


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))


if __name__ == "__main__":
    sys.exit(main())
