"""Builds the C-ABI shared library ``hot_b200/lib/libhot_b200.so`` with nvcc for sm_100a, and the torch
binding over it, ``hot_b200/lib/hot_torch.so``, with the host compiler.

    python -m hot_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU, so this also runs on a CPU-only machine.  The library
links the CUDA runtime statically and resolves the one driver entry point it needs
(cuTensorMapEncodeTiled) at run time, so it loads with ``dlopen`` on a machine without a
driver too (every entry point then fails with HOT_ERR_CUDA instead of computing).
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libhot_b200.so")
BINDING_PATH = os.path.join(LIB_DIR, "hot_torch.so")
SOURCES = ["common.cu", "status.cu", "row_ht_quant.cu", "col_ht_quant.cu", "go_dual.cu", "go_dual_tc.cu", "gemm_i8.cu", "linear.cu", "layer.cu",
           "conv.cu", "quant_tiles.cu", "quant_tiles_f32.cu", "gemm_grouped.cu", "gemm_conv.cu"]
BINDING_SOURCE = "torch_binding.cpp"
NVCC_FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "-Xcompiler", "-fPIC", "--cudart", "static"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def _stale() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(BINDING_PATH):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(BINDING_PATH))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", "hot_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def _binding_compile_command(obj: str) -> list:
    import sysconfig

    import torch
    root = os.path.join(os.path.dirname(torch.__file__), "include")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(ROOT, "include"), root, os.path.join(root, "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
           sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
            *["-I" + d for d in inc], "-c", os.path.join(CSRC, BINDING_SOURCE), "-o", obj]


def _binding_link_command(obj: str) -> list:
    import torch
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    return [os.environ.get("CXX", "g++"), "-shared", obj, "-o", BINDING_PATH, "-L" + libs, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
            "-ltorch", "-ltorch_python", "-L" + LIB_DIR, "-l:libhot_b200.so", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every source into objects (in parallel) and link the two shared libraries."""
    if not force and not _stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = _nvcc()
    inc = ["-I" + os.path.join(ROOT, "include"), "-I" + CSRC]
    procs = []
    for src in SOURCES:
        obj = os.path.join(obj_dir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, *inc, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    binding_obj = os.path.join(obj_dir, BINDING_SOURCE.replace(".cpp", ".o"))
    procs.append((BINDING_SOURCE, binding_obj, subprocess.Popen(_binding_compile_command(binding_obj), stdout=subprocess.PIPE,
                                                                stderr=subprocess.STDOUT, text=True)))
    objs = []
    for src, obj, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError("compilation of %s failed:\n%s" % (src, out))
        if verbose and out:
            print(out)
        if obj != binding_obj:
            objs.append(obj)
    cmd = [nvcc, "-shared", "--cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *objs]
    for link in (cmd, _binding_link_command(binding_obj)):
        r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
