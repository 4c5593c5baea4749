"""Builds the CUDA library ``libddhdg_b200.so`` in-tree for sm_100a."""

import os
import signal
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libddhdg_b200.so")
# translation units, compiled side by side: (source, extra flags)
UNITS = [("hdg_capi.cu", []), ("hdg_ndsolve.cu", [])] + \
    [(s, [f"-DDDHDG_DIM={d}"]) for s in ("hdg_condense_dim.cu", "hdg_batch_dim.cu") for d in (2, 3, 1)]
HEADER = os.path.join(HERE, "..", "include", "ddhdg_b200.h")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def nvcc():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def needs_build():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    return any(os.path.getmtime(d) > t for d in deps + [HEADER])


def build(force=False, verbose=False):
    if not force and not needs_build():
        return LIB
    with tempfile.TemporaryDirectory() as tmp:
        objs, jobs = [], []
        for i, (s, extra) in enumerate(UNITS):
            objs.append(os.path.join(tmp, f"{i}_{s}.o"))
            cmd = [nvcc()] + NVCC_FLAGS + extra + ["-c", "-o", objs[-1], os.path.join(CSRC, s)]
            if verbose:
                print(" ".join(cmd), file=sys.stderr)
            jobs.append((cmd, subprocess.Popen(cmd, start_new_session=True)))
        try:
            for cmd, job in jobs:
                if job.wait():
                    raise subprocess.CalledProcessError(job.returncode, cmd)
        finally:
            # after a failure: no compiler (nvcc and the programs it runs) may
            # outlive the directory it writes to
            for _, job in jobs:
                if job.poll() is None:
                    os.killpg(job.pid, signal.SIGTERM)
                job.wait()
        cmd = [nvcc()] + NVCC_FLAGS + ["-shared", "-o", LIB] + objs + ["-lcusolver", "-lcusparse"]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
