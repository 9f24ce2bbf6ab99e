"""In-tree build of libtlcuda.so for sm_100a with nvcc (no JIT cache, no torch).

``python -m torchlette_b200._build`` compiles every translation unit under
``csrc/`` to an object file (in parallel) and links the shared library next to
the sources, where the ctypes binding looks for it; ``tl_pycall.cpp`` becomes the
extension module ``_tlcall`` beside it, for the interpreter that builds it; without that interpreter's headers it is left out and
the calls go through ctypes.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(CSRC, "libtlcuda.so")
PYCALL = os.path.join(CSRC, "_tlcall" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = ["tl_api.cu", "tl_pool.cu", "tl_quantize.cu", "tl_qgemv.cu", "tl_qgemv_stream.cu", "tl_qgemm.cu", "tl_matmul.cu", "tl_matmul_tc.cu", "tl_elementwise.cu", "tl_decode_ops.cu", "tl_attention.cu", "tl_attention_tc.cu", "tl_int4.cu", "tl_autotune.cu", "tl_comm.cu"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden", "-ccbin", "g++",
]


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "tlcuda.h"))
    objs = []
    jobs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(CSRC, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [NVCC, *FLAGS, "-c", s, "-o", o]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0 or verbose:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"{os.path.basename(cmd[0])} failed for {cmd[-3] if cmd[0] == NVCC else cmd[-1]}")

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            list(ex.map(run, jobs))
    if jobs or _stale(LIB, objs):
        run([NVCC, "-shared", "-o", LIB, *objs, "-cudart", "static", "-ldl"])
    pysrc = os.path.join(CSRC, "tl_pycall.cpp")
    include = sysconfig.get_paths()["include"]
    if not os.path.exists(os.path.join(include, "Python.h")):
        sys.stderr.write(f"{include} has no Python.h: {os.path.basename(PYCALL)} is not built, calls go through ctypes\n")
    elif force or _stale(PYCALL, [pysrc, headers[-1]]):
        run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-I", include, "-o", PYCALL, pysrc])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
