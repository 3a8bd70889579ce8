"""Builds libxg_sm100.so (the C-ABI kernel library) in-tree with nvcc for sm_100a, and libxg_sm100_torch.so (the torch
operators on top of it) with the host compiler.

Usage: ``python -m xpu_graph_b200.build [--force] [--verbose]``.
Objects go to ``xpu_graph_b200/csrc/build/``; the shared libraries land next to this file so that they
travel with the source tree. Nothing here needs a GPU: nvcc cross-compiles.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(CSRC, "build")
LIB_PATH = os.path.join(HERE, "libxg_sm100.so")
TORCH_LIB_PATH = os.path.join(HERE, "libxg_sm100_torch.so")
TORCH_SOURCE = "torch_ops.cpp"
TORCH_STAMP = os.path.join(OBJ_DIR, "torch_ops.stamp")  # what the operators' library was built against

SOURCES = [
    "abi.cu",
    "norm.cu",
    "elementwise.cu",
    "copy_fusions.cu",
    "gemm.cu",
    "gemm_tc.cu",
    "gemm_tc_ksplit.cu",
    "gemm_mlp.cu",
    "mlp_small.cu",
    "gemm_f32.cu",
    "split_bf16x3.cu",
    "pad_rows.cu",
    "sdpa.cu",
    "sum3d.cu",
    "rowsum_cat.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++20", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; set NVCC or put it on PATH")
    return cand


def torch_abi() -> str:
    """What the operators' library has to agree on with the process that loads it."""
    import sysconfig

    import torch

    return f"torch {torch.__version__}, C++11 ABI {int(torch._C._GLIBCXX_USE_CXX11_ABI)}, {sysconfig.get_config_var('SOABI')}"


def _torch_stamp() -> str:
    import torch

    # (the library's run path names torch's folder)
    return f"{torch_abi()}\n{os.path.dirname(torch.__file__)}\n{os.environ.get('CXX', 'g++')}\n"


def _read_stamp() -> str:
    try:
        with open(TORCH_STAMP) as f:
            return f.read()
    except OSError:
        return ""


def built_for() -> str:
    """torch_abi() of the build, empty when that is not known."""
    return _read_stamp().split("\n")[0]


def _cuda_home() -> str:
    return os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))


def _compile_torch_ops(src: str, obj: str) -> str:
    import sysconfig

    import torch

    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"), "-isystem", sysconfig.get_paths()["include"],
           "-isystem", os.path.join(_cuda_home(), "include"), "-c", src, "-o", obj]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed for {src}:\n{proc.stdout}\n{proc.stderr}")
    return ""


def _link(cmd) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"link failed:\n{proc.stdout}\n{proc.stderr}")


def _deps_mtime() -> float:
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    paths.append(os.path.join(HERE, "..", "include", "xg_sm100.h"))
    paths.append(os.path.abspath(__file__))
    return max(os.path.getmtime(p) for p in paths)


def _compile_one(nvcc: str, src: str, obj: str, verbose: bool) -> str:
    cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{proc.stdout}\n{proc.stderr}")
    return proc.stderr if verbose else ""


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every source and link the two shared libraries. Returns the kernel library's path."""
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdr_time = _deps_mtime()

    def job(name):
        src, obj = os.path.join(CSRC, name), os.path.join(OBJ_DIR, os.path.splitext(name)[0] + ".o")
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_time)
        return src, obj, stale

    kernels = [job(name) for name in SOURCES]
    torch_src, torch_obj, torch_stale = job(TORCH_SOURCE)
    torch_stale = torch_stale or _read_stamp() != _torch_stamp()
    with cf.ThreadPoolExecutor(max_workers=8) as pool:
        futs = [pool.submit(_compile_torch_ops, torch_src, torch_obj)] if torch_stale else []
        futs += [pool.submit(_compile_one, nvcc, s, o, verbose) for s, o, stale in kernels if stale]
        for f in futs:
            out = f.result()
            if out:
                print(out, file=sys.stderr)
    if any(stale for _, _, stale in kernels) or not os.path.exists(LIB_PATH):
        _link([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *[o for _, o, _ in kernels]])
    if torch_stale or not os.path.exists(TORCH_LIB_PATH):
        import torch

        torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
        # The C++ runtime by its file name: a compiler that finds no libstdc++.so of its own takes libstdc++.a without a word, and
        # streams that cross between that copy and libtorch's end the process (an error message with a number in it did).
        _link([os.environ.get("CXX", "g++"), "-shared", "-o", TORCH_LIB_PATH, torch_obj, f"-L{HERE}", "-l:libxg_sm100.so", "-Wl,-rpath,$ORIGIN",
               f"-L{torch_lib}", f"-Wl,-rpath,{torch_lib}", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python",
               "-l:libstdc++.so.6"])
        with open(TORCH_STAMP, "w") as f:
            f.write(_torch_stamp())
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
