"""In-tree build of libdvm_b200.so (host JIT + sm_100a device interpreters + C ABI) and of the extension module _calls.

Usage: ``python -m dvm_b200.build [--force]``.  Needs nvcc (CUDA >= 12.8) and g++; cross-compiles for
sm_100a without a GPU.  _calls also takes Python's C headers; without them the package works through ctypes alone.  The shared library lands in ``dvm_b200/lib/`` next to the package so that it
travels with the source tree; nothing is installed outside the tree.
"""
import ctypes
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libdvm_b200.so")

CALLS_PATH = os.path.join(LIB_DIR, "_calls" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))

SOURCES = [
    "dvm_api.cc",
    "normalize.cc",
    "vcompile.cc",
    "vkernel.cc",
    "partition.cc",
    "stat_fusion.cc",
    "row_match.cc",
    "comm.cc",
    "runtime.cu",
    "staging.cc",
    "capi.cu",
    "vm_vector.cu",
    "vm_row.cu",
    "vm_stats.cu",
    "vm_direct.cu",
    "mm_tcgen05.cu",
    "mm_tile.cu",
    "attn_tcgen05.cu",
    "attn_decode.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    # the interpreters dispatch through dense switches: let ptxas build jump tables (the default threshold
    # of 101 % never does)
    "--jump-table-density=20",
    "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall,-Wno-unused-function",
]
# extra nvcc flags for experiments, e.g. DVM_B200_NVCC_EXTRA="--jump-table-density=101" (later flags win)
NVCC_FLAGS += os.environ.get("DVM_B200_NVCC_EXTRA", "").split()


def _nvcc():
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    path = os.path.join(cuda_home, "bin", "nvcc")
    return path if os.path.exists(path) else "nvcc"


def _newer(src, dst):
    return not os.path.exists(dst) or os.path.getmtime(src) > os.path.getmtime(dst)


def _loads(path):
    """False for a file that the loader refuses: cut short, or of another machine."""
    try:
        ctypes.CDLL(path)
    except OSError:
        return False
    return True


def _deps_mtime():
    latest = 0.0
    for d in (CSRC, os.path.join(HERE, "..", "include")):
        for f in os.listdir(d):
            if f.endswith((".h", ".cuh")):
                latest = max(latest, os.path.getmtime(os.path.join(d, f)))
    return latest


def build(force=False, verbose=False):
    os.makedirs(LIB_DIR, exist_ok=True)
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    hdr_time = _deps_mtime()
    jobs = []
    objs = []
    for src in SOURCES:
        sp = os.path.join(CSRC, src)
        op = os.path.join(obj_dir, src.rsplit(".", 1)[0] + ".o")
        objs.append(op)
        if force or _newer(sp, op) or hdr_time > os.path.getmtime(op):
            cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-x", "cu", "-c", sp, "-o", op]
            jobs.append(cmd)

    def run(cmd):
        try:
            r = subprocess.run(cmd, capture_output=True, text=True)
        except OSError as e:
            raise RuntimeError("build failed: %s: %s" % (cmd[0], e))
        if r.returncode != 0:
            raise RuntimeError("build failed: %s\n%s\n%s" % (" ".join(cmd), r.stdout, r.stderr))
        if verbose:
            sys.stderr.write(r.stderr)
        return r

    calls_src = os.path.join(CSRC, "py_calls.cc")
    calls_new = CALLS_PATH + ".new"   # (takes its place whole, or not at all)
    calls_job = force or _newer(calls_src, CALLS_PATH) or hdr_time > os.path.getmtime(CALLS_PATH) or not _loads(CALLS_PATH)

    def build_calls():   # (the front-end's calls into the C ABI; no CUDA in it)
        try:
            run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-Wall", "-Wno-missing-field-initializers",
                 "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(HERE, "..", "include"), calls_src, "-o", calls_new])
            os.replace(calls_new, CALLS_PATH)
        except RuntimeError as e:
            if os.path.exists(CALLS_PATH):   # (one of other sources)
                os.remove(CALLS_PATH)
            sys.stderr.write("dvm_b200: without the extension module _calls, which takes Python's C headers, a serving loop's steps go "
                             "through ctypes: slower, with the same results.  %s\n" % e)

    with ThreadPoolExecutor(max_workers=8) as ex:
        calls = [ex.submit(build_calls)] if calls_job else []
        list(ex.map(run, jobs))
        for f in calls:
            f.result()
    if jobs or not os.path.exists(LIB_PATH):
        run([_nvcc(), "-shared", "-o", LIB_PATH] + objs + ["-lcudart", "-ldl"])
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
