"""Build libmlb200.so (the C-ABI library) in-tree for sm_100a with nvcc.

    python -m maglua_b200.build          # or maglua_b200.build.build()
"""
import os
import shutil
import subprocess
import sys
import time

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmlb200.so")
# the long ones first
SOURCES = ["conv_fast.cu", "mx_f64.cu", "mx_f64_big.cu", "mx_f32.cu", "mx_f32_big.cu", "yzls_f32.cu", "yzls_f64.cu",
           "xstep_32.cu", "xstep_64.cu", "xstep_128.cu", "xstep_256.cu", "xstep_512.cu", "kernels.cu", "surrogate.cu",
           "capi.cu", "ewald.cu", "mx.cu", "yzls.cu"]
HEADERS = ["device.cuh", "fftreg.cuh", "fused.cuh", "kparams.h", "launch.h", "mx.cuh", "mxradix.h", "terms.cuh", "umma.cuh",
           "xreg.cuh", "xstep.cuh", "yzls.cuh"]

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-O2",
         "-I", os.path.join(ROOT, "include"), "-I", CSRC]


def _lineinfo(src):
    """Line tables, for profiles: three quarters of the size of the units that
    hold many instances of one kernel, and most of the time their modules take
    to load (mlb_init 230 ms with them), so there only on request."""
    many = src.startswith(("xstep_", "mx_f", "yzls_f"))
    return ["-lineinfo"] if not many or os.environ.get("MLB_LINEINFO") else []


def nvcc():
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS]
    deps.append(os.path.join(ROOT, "include", "mlb200.h"))
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force=False, verbose=False):
    """Compile every .cu into one shared library (static cudart)."""
    if not force and not _stale():
        return LIB
    objs, running = [], []
    jobs = max(1, os.cpu_count() or 1)
    bdir = os.path.join(HERE, "_build")
    os.makedirs(bdir, exist_ok=True)
    for src in SOURCES:   # side by side, one per core
        obj = os.path.join(bdir, src.replace(".cu", ".o"))
        cmd = [nvcc()] + ARCH + FLAGS + _lineinfo(src) + ["-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd))
        while sum(p.poll() is None for _, p in running) >= jobs:
            time.sleep(0.05)
        running.append((cmd, subprocess.Popen(cmd)))
        objs.append(obj)
    failed = [cmd for cmd, p in running if p.wait() != 0]
    if failed:
        raise subprocess.CalledProcessError(1, failed[0])
    tmp = LIB + ".tmp"
    subprocess.check_call([nvcc()] + ARCH + ["-shared", "-o", tmp] + objs + ["-lcudart_static", "-lrt", "-ldl", "-lpthread"])
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
