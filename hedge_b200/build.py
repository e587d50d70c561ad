"""Builds libhedge_b200.so (sm_100a) in-tree with nvcc.

The shared library sits next to this file so that it travels with the
source tree; ``python -m hedge_b200.build`` rebuilds it.
"""

from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libhedge_b200.so")
SOURCES = ["api.cu", "rhs_simt.cu", "rhs_split.cu", "norm.cu", "adjoint.cu", "ensemble.cu",
           "waitcheck.cu", "rhs_quad.cu", "quad_fp64.cu"]
# the FP64 tensor-core kernels' instances, in parts that compile side by side:
# (source, macro that selects the part, parts)
PARTS = [("rhs_fp64.cu", "HB_FP64_PART", 5), ("adjoint_fp64.cu", "HB_ADJ_PART", 4)]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def needs_rebuild():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(HERE, "..", "include", "hedge_b200.h"))
    return any(os.path.getmtime(p) > t for p in deps if os.path.exists(p))


def build(force=False, verbose=False, extra_flags=()):
    if not force and not needs_rebuild():
        return LIB
    objs = []
    build_dir = os.path.join(HERE, "_build")
    os.makedirs(build_dir, exist_ok=True)
    procs = []
    units = [(src, src.replace(".cu", ".o"), []) for src in SOURCES]
    units += [(src, src.replace(".cu", "_%d.o" % p), ["-D%s=%d" % (macro, p)])
              for src, macro, n in PARTS for p in range(n)]
    for src, obj, defines in units:
        obj = os.path.join(build_dir, obj)
        cmd = [nvcc(), "-std=c++17", "-O3", *ARCH, "-lineinfo", "-Xcompiler", "-fPIC",
               "-Xptxas", "-v" if verbose else "-O3", "--expt-relaxed-constexpr",
               *extra_flags, *defines, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE,
                                            stderr=subprocess.STDOUT)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            sys.stderr.write(out.decode())
            raise RuntimeError("nvcc failed on %s" % src)
        if verbose:
            sys.stderr.write(out.decode())
    tmp = LIB + ".tmp"
    subprocess.check_call([nvcc(), "-shared", *ARCH, "-o", tmp, *objs,
                           "-Xcompiler", "-fPIC"])
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
