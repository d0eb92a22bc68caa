"""Compiles the CUDA sources of this directory into libci_b200.so (sm_100a only) and the host extension
host.cpp into _ci_host.so, which is linked against it.

    python comp_inference_b200/csrc/build.py [--force] [--verbose]

The library is built in-tree, next to the sources, and is the only thing the
Python package loads; there is no other backend.
"""
import argparse
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libci_b200.so")
HOST_SRC = os.path.join(HERE, "host.cpp")
HOST = os.path.join(HERE, "_ci_host.so")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def sources():
    return sorted(glob.glob(os.path.join(HERE, "*.cu")))


def _deps():
    return sources() + glob.glob(os.path.join(HERE, "*.cuh")) + [
        os.path.join(os.path.dirname(os.path.dirname(HERE)), "include", "comp_inference_b200.h")]


def stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(p) > t for p in _deps())


def host_stale():
    if not os.path.exists(HOST):
        return True
    t = os.path.getmtime(HOST)
    return any(os.path.getmtime(p) > t for p in (HOST_SRC, os.path.join(
        os.path.dirname(os.path.dirname(HERE)), "include", "comp_inference_b200.h")))


def start_host():
    """Starts the compiler on host.cpp; returns (process, object file)."""
    import sysconfig
    import torch
    root = os.path.join(os.path.dirname(torch.__file__))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")]
    obj = HOST_SRC[:-4] + ".o"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-c", HOST_SRC, "-o", obj, "-DTORCH_API_INCLUDE_EXTENSION_H",
           "-DTORCH_EXTENSION_NAME=_ci_host", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for d in inc:
        cmd += ["-isystem", d]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True), obj


def link_host(obj):
    import torch
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    subprocess.check_call(["g++", "-shared", obj, "-o", HOST, LIB, f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu",
                           "-ltorch_python", "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{lib}"])
    os.remove(obj)


def build(force=False, verbose=False):
    host = start_host() if force or host_stale() else None
    if not force and not stale():
        return finish_host(host)
    objs = []
    procs = []
    for src in sources():
        obj = src[:-3] + ".o"
        cmd = ["nvcc", "-O3", "-std=c++17", *ARCH, "-lineinfo", "-Xcompiler", "-fPIC", "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {os.path.basename(src)}\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.check_call(["nvcc", "-shared", *ARCH, *objs, "-o", LIB, "-lcudart", "-Xlinker", "-soname=libci_b200.so"])
    for o in objs:
        os.remove(o)
    return finish_host(host)


def finish_host(host):
    if host is not None:
        out, _ = host[0].communicate()
        if host[0].returncode != 0:
            sys.stderr.write(f"--- host.cpp\n{out}\n")
            raise RuntimeError("g++ failed")
        link_host(host[1])
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
