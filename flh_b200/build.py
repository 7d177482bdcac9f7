"""Build libflh_b200.so (sm_100a only) in-tree with nvcc.

    python -m flh_b200.build          # or: from flh_b200.build import build; build()

The library has no Python or torch dependency: it is the C ABI declared in
include/flh_b200.h.  nvcc cross-compiles without a GPU.  The Python extension beside it
(csrc/host_calls.cpp) needs torch, a C++ compiler and CPython's headers; where it cannot be
built the build says so and goes on, and flh_b200/_CUDA.py does without it.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SOURCES = ["api.cu", "quant_group.cu", "quant_token.cu", "quant_token_warp.cu", "quant_token_factor.cu", "quant_token_tc.cu", "act.cu", "gemm_mma.cu", "gemm_tcgen05.cu", "gemm_i8.cu", "gemm_group_f8.cu", "gemm_decode_tc.cu", "gemm_decode_ring.cu", "gptq.cu", "allreduce.cu"]
LIB = os.path.join(HERE, "libflh_b200.so")
# csrc/host_calls.cpp: the per-call host work as a Python extension.  It is compiled against one CPython (the file's suffix) and one
# torch, whose version is kept beside the objects and in the extension itself.
HOST = os.path.join(HERE, "_host" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
HOST_TORCH = os.path.join(HERE, "build", "_host.torch")
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(verbose: bool = False, force: bool = False) -> str:
    nvcc = os.environ.get("NVCC", "nvcc")
    headers = [os.path.join(CSRC, "common.cuh"), os.path.join(CSRC, "token_common.cuh"), os.path.join(CSRC, "tc_common.cuh"), os.path.join(CSRC, "tc_pair.cuh"), os.path.join(CSRC, "act_common.cuh"), os.path.join(CSRC, "tc_quant_common.cuh"), os.path.join(HERE, "..", "include", "flh_b200.h")]
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", s, "-o", o] + (["-Xptxas", "-v"] if verbose else [])
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0 or verbose:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"{cmd[0]} failed for {cmd[cmd.index('-o') + 1]}")

    with ThreadPoolExecutor(max_workers=min(4, max(1, len(jobs)))) as ex:
        list(ex.map(run, jobs))
    if force or jobs or not os.path.exists(LIB):
        run([nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"])
    try:
        _build_host(run, force)
    except (ImportError, OSError, RuntimeError) as e:
        warnings.warn(f"flh_b200._host was not built, small calls take twice the host time: {e}")
    return LIB


def _build_host(run, force: bool) -> None:
    import torch
    src = os.path.join(CSRC, "host_calls.cpp")
    if not force and not _stale(HOST, [src, os.path.join(HERE, "..", "include", "flh_b200.h")]) and _built_for() == torch.__version__:
        return
    if os.path.exists(HOST):
        os.remove(HOST)                             # what does not build again is not loaded
    from torch.utils import cpp_extension
    if torch.version.cuda is None:
        return                                      # nothing to launch on: flh_b200/_CUDA.py does without
    include = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cpp_extension.CUDA_HOME or "/usr/local/cuda", "include")]
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DFLH_TORCH="{torch.__version__}"',
         *[f"-I{i}" for i in include], src, "-o", HOST, f"-L{torch_lib}", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-ltorch_cuda",
         "-ltorch_python", f"-L{HERE}", "-l:libflh_b200.so", "-Wl,-rpath,$ORIGIN"])
    with open(HOST_TORCH, "w") as f:
        f.write(torch.__version__)


def _built_for():
    """The torch version that HOST was compiled against, or None."""
    try:
        with open(HOST_TORCH) as f:
            return f.read()
    except OSError:
        return None


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
