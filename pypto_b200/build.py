"""In-tree build of libdsv32_b200.so with nvcc for sm_100a, and of the native front end _front.so with g++.

    python -m pypto_b200.build [--verbose] [--force]

Both are written next to this file (pypto_b200/libdsv32_b200.so, pypto_b200/_front.so) so that they ship
with a source snapshot of the tree; nothing is installed anywhere else.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_NAME = "libdsv32_b200.so"
LIB_PATH = os.path.join(HERE, LIB_NAME)
SOURCES = ["api.cu", "topk.cu", "indexer_tc.cu", "sfa_tc.cu", "scfa_tc.cu", "sfa_combine.cu", "gemm_tc.cu", "heads_tc.cu", "prolog_finish.cu", "prolog_v4.cu", "v4_q_tc.cu", "pg_prolog.cu",
           "mla_prolog_v4.cu", "hc_pre.cu", "hc_pre_tc.cu", "compressor.cu", "decode_advance.cu", "noalloc.cu"]
FRONT_SOURCE, FRONT_PATH = os.path.join(CSRC, "front.cpp"), os.path.join(HERE, "_front.so")
FRONT_TORCH = os.path.join(HERE, "build", "front_torch")   # the torch release _front.so was linked against
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc_path() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return cand


def _sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _newest_source_mtime() -> float:
    m = 0.0
    for root in (CSRC, os.path.join(os.path.dirname(HERE), "include")):
        for f in os.listdir(root):
            m = max(m, os.path.getmtime(os.path.join(root, f)))
    return m


def is_stale() -> bool:
    newest = _newest_source_mtime()
    return any(not os.path.exists(p) or os.path.getmtime(p) < newest for p in (LIB_PATH, FRONT_PATH)) or not _front_fits_torch()


def _front_fits_torch() -> bool:
    import torch
    try:
        with open(FRONT_TORCH) as f:
            return f.read() == torch.__version__
    except OSError:
        return False


def _front_command() -> list:
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(nvcc_path()))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[f"-I{i}" for i in inc], FRONT_SOURCE, "-o", FRONT_PATH, f"-L{os.path.join(root, 'lib')}", "-ltorch_python",
            "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def build(verbose: bool = False, force: bool = False) -> str:
    if not force and not is_stale():
        return LIB_PATH
    objs = []
    build_dir = os.path.join(HERE, "build")
    os.makedirs(build_dir, exist_ok=True)
    common = [nvcc_path(), *ARCH_FLAGS, "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC",
              "--expt-relaxed-constexpr"]
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    for src in _sources():
        obj = os.path.join(build_dir, os.path.basename(src) + ".o")
        objs.append(obj)
        procs.append((src, subprocess.Popen(common + ["-c", src, "-o", obj], stdout=subprocess.PIPE,
                                            stderr=subprocess.STDOUT, text=True)))
    procs.append((FRONT_SOURCE, subprocess.Popen(_front_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0 or verbose:
            sys.stderr.write(f"--- {os.path.basename(src)} ---\n{out}\n")
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("nvcc or g++ failed; see output above")
    import torch
    with open(FRONT_TORCH, "w") as f:
        f.write(torch.__version__)
    link = [nvcc_path(), *ARCH_FLAGS, "-shared", "-o", LIB_PATH, *objs, "-lcudart"]
    res = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if res.returncode != 0:
        raise RuntimeError("link failed:\n" + res.stdout)
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--force", action="store_true")
    a = ap.parse_args()
    print(build(verbose=a.verbose, force=a.force))
