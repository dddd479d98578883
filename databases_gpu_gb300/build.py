"""Build libdycuckoo.so in-tree with nvcc for sm_103a (GB300).

The library is plain C ABI (include/dycuckoo.h): no torch types cross it.
Translation units compile in parallel; nothing is rebuilt when the shared
object is newer than every source and header.
"""
from __future__ import annotations

import os
import shutil
import subprocess

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
BUILD_DIR = os.path.join(ROOT, "_build")
LIB = os.path.join(PKG, "libdycuckoo.so")

SOURCES = ["dyc_ops4.cu", "dyc_ops8.cu", "dyc_bins4.cu", "dyc_bins8.cu",
           "dyc_api.cu", "dyc_server.cu"]
# one module per key width and bucket size: a process loads those it uses
SOURCES += [("dyc_bins_sb.cu", kb, sb) for kb in (4, 8) for sb in (32, 64, 128)]
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
# Device code uncompressed: unpacking it took 10 ms of the first use of a key
# width's bin kernels (0.8 without); the library is 38 MB for it.
NVCC_FLAGS = ARCH + ["--compress-mode=none", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
                     "-I", INCLUDE, "-I", CSRC]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the DyCuckoo CUDA library cannot be built")


def _inputs():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    files += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return [f for f in files if f.endswith((".cu", ".cuh", ".h", ".hpp"))]


def up_to_date(lib: str = LIB) -> bool:
    if not os.path.exists(lib):
        return False
    t = os.path.getmtime(lib)
    return all(os.path.getmtime(f) <= t for f in _inputs())


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    os.makedirs(BUILD_DIR, exist_ok=True)
    cc = nvcc()
    procs = []
    objs = []
    for src in SOURCES:
        name, defs = src, []
        if not isinstance(src, str):
            src, kb, sb = src
            name, defs = "dyc_bins_sb%d_%d.cu" % (kb, sb), ["-DDYC_KB=%d" % kb, "-DDYC_SB=%d" % sb]
        obj = os.path.join(BUILD_DIR, name.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [cc] + NVCC_FLAGS + defs + ["-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            print(" ".join(cmd))
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE,
                                            stderr=subprocess.STDOUT)))
    for cmd, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError("nvcc failed (%s):\n%s" % (" ".join(cmd), out.decode(errors="replace")))
    tmp = LIB + ".tmp%d" % os.getpid()
    cmd = [cc] + ARCH + ["-shared", "-cudart", "shared", "-o", tmp] + objs
    if verbose:
        print(" ".join(cmd))
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n%s" % r.stdout.decode(errors="replace"))
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force=True, verbose=True))
