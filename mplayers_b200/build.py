"""Builds libmplayers_b200.so (the C-ABI library with the sm_100a kernels) in-tree with nvcc.

    python -m mplayers_b200.build [--force] [--verbose]
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmplayers_b200.so")
SOURCES = ["mp_api.cu", "mp_forward.cu", "mp_fwd_tma.cu", "mp_fwd_tma_rank1.cu", "mp_fwd_tma_stride.cu", "mp_backward.cu", "mp_wide.cu", "mp_wide_train.cu", "mp_wide_team.cu",
           "mp_wide_many.cu", "mp_pair_rows.cu", "mp_wide_bwd.cu", "mp_bwd_quad.cu", "mp_soft.cu", "mp_soft_cta.cu", "mp_terms.cu", "mp_swbp.cu"]
HEADERS = [os.path.join(CSRC, "mp_common.cuh"), os.path.join(CSRC, "mp_minplus.cuh"), os.path.join(CSRC, "mp_wide.cuh"),
           os.path.join(CSRC, "mp_fwd_tma.cuh"),
           os.path.join(os.path.dirname(HERE), "include", "mplayers_b200.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--use_fast_math=false"]


def _nvcc():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    flags = [f for f in NVCC_FLAGS if f != "--use_fast_math=false"]
    if verbose:
        flags += ["-Xptxas", "-v"]
    objs = []
    procs = []
    for s in SOURCES:
        src = os.path.join(CSRC, s)
        obj = os.path.join(CSRC, s.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [src] + HEADERS):
            procs.append((s, subprocess.Popen([_nvcc()] + flags + ["-c", src, "-o", obj],
                                              stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    for s, p in procs:
        out = p.communicate()[0].decode()
        if p.returncode != 0:
            raise RuntimeError("nvcc failed on %s:\n%s" % (s, out))
        if verbose:
            print(out)
    if force or procs or _stale(LIB, objs):
        subprocess.check_call([_nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
