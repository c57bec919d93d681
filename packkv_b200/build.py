"""Builds packkv_b200/libpackkv_sm100.so (the kernels and the C ABI, nvcc for sm_100a) and packkv_b200/_host.so (the host
path of packkv_b200.ops, a CPython extension over torch's tensors) in-tree.

    python -m packkv_b200.build [--force]

The shared library is the product's only compute path; nothing falls back to the CPU.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libpackkv_sm100.so")
SOURCES = ["pack.cu", "quant.cu", "attn.cu", "legacy.cu", "cache.cu", "dense.cu", "reorder.cu", "fused_encode.cu", "encode_entry.cu", "capi.cu"]
HOST_SOURCE = os.path.join(CSRC, "host.cpp")
HOST_LIB = os.path.join(PKG, "_host.so")
HOST_STAMP = os.path.join(OBJ, "_host.stamp")
HEADER = os.path.join(os.path.dirname(PKG), "include", "packkv_sm100.h")
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command():
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
               sysconfig.get_paths()["include"]]
    lib = os.path.join(root, "lib")
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
            + [x for i in include for x in ("-isystem", i)] + [HOST_SOURCE, "-o", HOST_LIB]
            + [f"-L{lib}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10_cuda", "-lc10"])


def _host_key() -> str:
    """What _host.so was built with and against: it shares the layout of torch's and CPython's classes."""
    import sysconfig

    import torch
    return "\n".join([torch.__version__, str(sysconfig.get_config_var("SOABI"))] + _host_command())


def _host_stale() -> bool:
    if _stale(HOST_LIB, [HOST_SOURCE, HEADER]) or not os.path.exists(HOST_STAMP):
        return True
    with open(HOST_STAMP) as f:
        return f.read() != _host_key()


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(HEADER)
    jobs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src.replace(".cu", ".o"))
        if force or _stale(o, [s] + headers):
            jobs.append((s, o))

    def compile_one(job):
        if job is None:
            r = subprocess.run(_host_command(), capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"g++ failed for {HOST_SOURCE}:\n{r.stdout}\n{r.stderr}")
            with open(HOST_STAMP, "w") as f:
                f.write(_host_key())
            return
        s, o = job
        r = subprocess.run([_nvcc()] + NVCC_FLAGS + ["-c", s, "-o", o], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {s}:\n{r.stdout}\n{r.stderr}")
        with open(o + ".ptxas.txt", "w") as f:
            f.write(r.stderr)
        if verbose:
            print(r.stderr)

    host = [None] if force or _host_stale() else []
    with ThreadPoolExecutor(max_workers=8) as pool:
        list(pool.map(compile_one, jobs + host))
    objs = [os.path.join(OBJ, s.replace(".cu", ".o")) for s in SOURCES]
    if force or jobs or _stale(LIB, objs):
        r = subprocess.run([_nvcc(), "-shared", "-o", LIB] + objs, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
