"""Builds libflagattn_b200.so in-tree with nvcc for sm_100a.

Every .cu file under csrc/ is compiled to an object (in parallel, skipped when
the object is newer than all sources and headers) and linked into
flagattention_b200/lib/libflagattn_b200.so with the CUDA runtime linked
statically, so the library loads on a machine without a GPU or a CUDA
installation (symbol checks) and needs only the driver to run.
"""
import concurrent.futures
import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")
LIB_DIR = os.path.join(PKG_DIR, "lib")
OBJ_DIR = os.path.join(LIB_DIR, "obj")
LIB_PATH = os.path.join(LIB_DIR, "libflagattn_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "ops.cpp")
HOST_PATH = os.path.join(LIB_DIR, "flagattn_host.so")
HOST_STAMP = os.path.join(OBJ_DIR, "flagattn_host.command")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-I", INCLUDE, "-I", CSRC,
]

HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared"]
HOST_LIBS = ["-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", "-lflagattn_b200",
             "-Wl,-rpath,$ORIGIN"]


def _nvcc():
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found; cannot build libflagattn_b200.so")
    return path


def _sources():
    out = []
    for root, _, files in os.walk(CSRC):
        for f in sorted(files):
            if f.endswith(".cu"):
                out.append(os.path.join(root, f))
    return sorted(out)


def _headers_mtime():
    newest = 0.0
    for root, _, files in os.walk(CSRC):
        for f in files:
            if f.endswith((".cuh", ".h")):
                newest = max(newest, os.path.getmtime(os.path.join(root, f)))
    for f in os.listdir(INCLUDE):
        newest = max(newest, os.path.getmtime(os.path.join(INCLUDE, f)))
    return newest


def _compile_one(nvcc, src, obj, verbose):
    cmd = [nvcc] + NVCC_FLAGS + ["-c", src, "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, res.stdout, res.stderr))
    if verbose:
        print("compiled", os.path.relpath(src, PKG_DIR), flush=True)
    return obj


def build(force=False, verbose=False):
    """Compiles what is out of date and links the shared library. Returns its path."""
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdr_time = _headers_mtime()
    jobs, objs = [], []
    for src in _sources():
        rel = os.path.relpath(src, CSRC).replace(os.sep, "__")
        obj = os.path.join(OBJ_DIR, rel[:-3] + ".o")
        objs.append(obj)
        stale = (force or not os.path.exists(obj)
                 or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_time))
        if stale:
            jobs.append((src, obj))
    if jobs:
        workers = max(1, min(len(jobs), os.cpu_count() or 1))
        with concurrent.futures.ThreadPoolExecutor(workers) as pool:
            futs = [pool.submit(_compile_one, nvcc, s, o, verbose) for s, o in jobs]
            for f in futs:
                f.result()
    need_link = (jobs or not os.path.exists(LIB_PATH)
                 or any(os.path.getmtime(o) > os.path.getmtime(LIB_PATH) for o in objs))
    if need_link:
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a",
               "-cudart", "static", "-o", LIB_PATH] + objs
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("link failed:\n%s\n%s" % (res.stdout, res.stderr))
        if verbose:
            print("linked", LIB_PATH, flush=True)
    _build_host(force, verbose)
    return LIB_PATH


def host_tag():
    """What a build of the host extension is good for: it inlines torch's C++ headers, whose layouts hold for one release
    and one way of compiling only, and Python's own interface."""
    import sysconfig

    import torch
    return "torch %s, %s, cxx11 abi %d" % (torch.__version__, sysconfig.get_config_var("SOABI"),
                                           torch._C._GLIBCXX_USE_CXX11_ABI)


def _host_stamp():
    """What the extension on disk has to have been made for and with (no paths: a built tree may be moved)."""
    return host_tag() + "\n" + " ".join(HOST_FLAGS + HOST_LIBS)


def _host_current(header):
    if not os.path.exists(HOST_PATH) or not os.path.exists(HOST_STAMP):
        return False
    with open(HOST_STAMP) as f:
        if f.read() != _host_stamp():
            return False
    return os.path.getmtime(HOST_PATH) >= max(os.path.getmtime(HOST_SRC), os.path.getmtime(header))


def _build_host(force, verbose):
    """The operators' host side (csrc/host/ops.cpp), a Python extension on torch's C++ interface and the library."""
    if not force and _host_current(os.path.join(INCLUDE, "flagattn_b200.h")):
        return
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    fresh = HOST_PATH + ".new"
    cmd = (["g++"] + HOST_FLAGS
           + ["-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI, '-DFA_HOST_TAG="%s"' % host_tag(), "-I", INCLUDE,
              "-isystem", os.path.join(root, "include"),
              "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
              "-isystem", os.path.join(cuda, "include"), "-isystem", sysconfig.get_paths()["include"],
              HOST_SRC, "-o", fresh, "-L", os.path.join(root, "lib"), "-L", LIB_DIR] + HOST_LIBS)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed for %s:\n%s\n%s" % (HOST_SRC, res.stdout, res.stderr))
    os.replace(fresh, HOST_PATH)   # a process that has the old one loaded keeps it
    with open(HOST_STAMP, "w") as f:
        f.write(_host_stamp())
    if verbose:
        print("linked", HOST_PATH, flush=True)


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
