"""Builds libpicasso_b200.so from csrc/*.cu with nvcc for sm_100a, and the torch extension _torch_ops.so (the native
host path over the library's C ABI) from csrc/torch_ops.cpp with g++, in-tree.

    python -m picassoplus_b200.build [--force] [--verbose]

Objects are rebuilt only when their source (or a header) is newer.  The library links the
CUDA runtime statically, exports the C ABI declared in include/picasso_b200.h, and
has no dependency on torch; the extension links the library and torch.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(PKG, "libpicasso_b200.so")
OPS = os.path.join(PKG, "_torch_ops.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


# Per-file flags.  The decimation kernels round every float operation on its own (no fused
# multiply-add) so that their edge costs, and with them the clustering, are reproducible by plain C.
FILE_FLAGS = {"decimate.cu": ["--fmad=false"], "f2f_tc_one.cu": ["-Xptxas", "-v"]}
# Registers per thread that kernels have to be built with: f2f_tc_one.cu deals out what its blocks are launched with, and its
# calls refuse a kernel that was built with fewer.
REGISTERS = {"f2f_tc_one.cu": ("f2f_one_sample_tc_kernel", 96)}


def wrong_registers(ptxas: str, kernel: str, count: int):
    """Lines of the assembler's report that give a kernel of this name another number of registers."""
    wrong, name = [], ""
    for line in ptxas.splitlines():
        if "Compiling entry function" in line:
            name = line
        elif "Used " in line and kernel in name and f"Used {count} registers" not in line:
            wrong.append(name + line)
    return wrong


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers_mtime() -> float:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(ROOT, "include", "picasso_b200.h"))
    return max(os.path.getmtime(h) for h in hs)


def _ops_command(out: str):
    """g++ command of the torch extension: torch's own headers, libraries and C++ ABI."""
    import sysconfig
    import torch
    t = os.path.join(os.path.dirname(torch.__file__))
    inc, lib = os.path.join(t, "include"), os.path.join(t, "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    return (["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_torch_ops",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] +
            [a for d in (inc, os.path.join(inc, "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
                         sysconfig.get_paths()["include"]) for a in ("-isystem", d)] +
            [os.path.join(CSRC, "torch_ops.cpp"), "-o", out, "-L" + PKG, "-l:libpicasso_b200.so", "-L" + lib, "-lc10", "-lc10_cuda",
             "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN:" + lib])


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    hm = _headers_mtime()
    jobs = []
    objs = []
    for src in sources():
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src[:-3] + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hm):
            cmd = [nvcc] + NVCC_FLAGS + FILE_FLAGS.get(src, []) + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    def check(cmd, r):
        if verbose or r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("build step failed: " + " ".join(cmd[-3:]))

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for cmd, r in ex.map(run, jobs):
                check(cmd, r)
                src = os.path.basename(cmd[-3])
                if src in REGISTERS and wrong_registers(r.stdout + r.stderr, *REGISTERS[src]):
                    os.remove(cmd[-1])
                    raise RuntimeError(f"{src}: {REGISTERS[src][0]} is not built with {REGISTERS[src][1]} registers:\n" +
                                       "\n".join(wrong_registers(r.stdout + r.stderr, *REGISTERS[src])))
    if jobs or not os.path.exists(LIB):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-cudart", "static",
               "-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    ops_src = os.path.join(CSRC, "torch_ops.cpp")
    if force or not os.path.exists(OPS) or os.path.getmtime(OPS) < max(os.path.getmtime(ops_src), hm):
        check(*run(_ops_command(OPS)))
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
