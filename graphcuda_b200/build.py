"""In-tree build of the C-ABI library ``lib/libgraphcuda_b200.so`` with nvcc.

Every translation unit is compiled for sm_100a only (``-gencode
arch=compute_100a,code=sm_100a``), without fast-math (the adjacency
normalisation must round like IEEE/torch-CPU), and linked into one shared
object with the static CUDA runtime.  The driver API is reached through
``cudaGetDriverEntryPoint`` at run time, so the library has no link-time
dependency on libcuda and builds on a machine without a GPU.

The native host side (``csrc/host/*.cpp``: torch tensors in, C-ABI calls out) is
compiled with g++ against the installed torch into ``lib/_gc_host.so``.

Usage:  python -m graphcuda_b200.build [-v] [--force]
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIBDIR = os.path.join(PKG, "lib")
OBJDIR = os.path.join(LIBDIR, "obj")
LIBNAME = "libgraphcuda_b200.so"

SOURCES = [
    "abi.cu",
    "spmm_csr.cu",
    "gather_probe.cu",
    "gemm.cu",
    "gemm_simt.cu",
    "gemm_narrow.cu",
    "gemm_tcgen05.cu",
    "elementwise.cu",
    "gcn_layer.cu",
    "graph_build.cu",
    "loss.cu", "optim.cu",
]

HOSTSRC = os.path.join(CSRC, "host")
HOSTNAME = "_gc_host"
HOST_SOURCES = ["core.cpp", "layer.cpp", "tail.cpp", "bind.cpp"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def lib_path() -> str:
    return os.path.join(LIBDIR, LIBNAME)


def host_path() -> str:
    return os.path.join(LIBDIR, HOSTNAME + ".so")


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")
    return cand


def _deps_mtime() -> float:
    t = 0.0
    for root in (CSRC, os.path.join(os.path.dirname(PKG), "include")):
        for f in os.listdir(root):
            if f.endswith((".cu", ".cuh", ".h")):
                t = max(t, os.path.getmtime(os.path.join(root, f)))
    return t


def _sources() -> list[str]:
    return [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _host_jobs(force: bool):
    """(compile jobs, object files) of the native host side."""
    import sysconfig

    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    flags = ["-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden", f"-DTORCH_EXTENSION_NAME={HOSTNAME}",
             "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
             "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"),
             "-isystem", os.path.join(cuda, "include"), "-isystem", sysconfig.get_paths()["include"]]
    headers = [os.path.join(HOSTSRC, "host.h"), os.path.join(os.path.dirname(PKG), "include", "graphcuda_b200.h")]
    newest_header = max(os.path.getmtime(h) for h in headers)
    jobs, objs = [], []
    for src in HOST_SOURCES:
        sp, op = os.path.join(HOSTSRC, src), os.path.join(OBJDIR, "host_" + src[:-4] + ".o")
        objs.append(op)
        if force or not os.path.exists(op) or os.path.getmtime(op) < max(os.path.getmtime(sp), newest_header):
            jobs.append((src, [os.environ.get("CXX", "g++"), *flags, "-c", sp, "-o", op]))
    return jobs, objs


def _link_host(objs) -> None:
    import torch
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-shared", "-o", host_path(), *objs, "-L" + libs, "-Wl,-rpath," + libs,
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-ldl",
           *_cudart_link()]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("host link failed:\n" + r.stdout + r.stderr)


def _cudart_link() -> list[str]:
    """The CUDA runtime torch itself uses (found through torch's own libraries at load time)."""
    lib64 = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "lib64")
    return ["-L" + lib64, "-lcudart"]


def build(verbose: bool = False, force: bool = False, ptxas_verbose: bool = False) -> str:
    """Compile what is out of date and link; returns the path of the C-ABI library."""
    os.makedirs(OBJDIR, exist_ok=True)
    nvcc = _nvcc()
    newest = _deps_mtime()
    headers_newest = max(
        [os.path.getmtime(os.path.join(CSRC, f)) for f in os.listdir(CSRC) if f.endswith(".cuh")]
        + [os.path.getmtime(os.path.join(os.path.dirname(PKG), "include", "graphcuda_b200.h"))]
    )
    jobs = []
    objs = []
    for src in _sources():
        sp = os.path.join(CSRC, src)
        op = os.path.join(OBJDIR, src[:-3] + ".o")
        objs.append(op)
        stale = force or not os.path.exists(op) or os.path.getmtime(op) < max(os.path.getmtime(sp), headers_newest)
        if stale:
            cmd = [nvcc, *NVCC_FLAGS, "-c", sp, "-o", op]
            if ptxas_verbose:
                cmd[1:1] = ["-Xptxas", "-v"]
            jobs.append((src, cmd))
    host_jobs, host_objs = _host_jobs(force)

    def run(job):
        src, cmd = job
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r.returncode, r.stdout + r.stderr

    if jobs or host_jobs:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs) + len(host_jobs))) as ex:
            for src, rc, out in ex.map(run, jobs + host_jobs):
                if verbose or rc != 0 or ptxas_verbose:
                    sys.stderr.write(f"[{src}] rc={rc}\n{out}\n")
                if rc != 0:
                    raise RuntimeError(f"compilation of {src} failed:\n{out}")
    lp = lib_path()
    if jobs or not os.path.exists(lp) or os.path.getmtime(lp) < newest:
        cmd = [nvcc, "-shared", "-o", lp, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    if host_jobs or not os.path.exists(host_path()):
        _link_host(host_objs)
    return lp


if __name__ == "__main__":
    p = build(verbose="-v" in sys.argv, force="--force" in sys.argv, ptxas_verbose="--ptxas" in sys.argv)
    print(p)
