"""Builds libkvcache_b200.so (sm_100a) from csrc/ with nvcc, in-tree.

Usage: python build.py [--force] [--verbose]
The shared library lands in lib/ beside this file. It links only the CUDA
runtime (statically) and libdl; NCCL is resolved with dlopen at first use.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIBDIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIBDIR, "libkvcache_b200.so")

SOURCES = [
    "memory.cu",
    "append.cu",
    "quantize.cu",
    "attn_general.cu",
    "attn_decode.cu",
    "attn_packed.cu",
    "attn_turbo.cu", "attn_turbo_v4.cu",
    "attn_f32.cu", "attn_stream.cu", "attn_stream_bf16_64.cu", "attn_stream_bf16_128.cu", "attn_stream_bf16_256.cu",
    "attn_stream_f16_64.cu", "attn_stream_f16_128.cu", "attn_stream_f16_256.cu",
    "attn_chunk_packed.cu", "attn_chunk_tc.cu", "attn_chunk_one_tc.cu", "attn_chunk_mat.cu", "attn_chunk_pairs.cu", "attn_verify_tc.cu",
    "attn_dispatch.cu",
    "cache.cu",
    "round.cu",
    "capi.cu",
    "promptcache.cu",
    "comm.cu",
    "noalloc.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=default",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _newer(src: str, dst: str, deps) -> bool:
    if not os.path.exists(dst):
        return True
    t = os.path.getmtime(dst)
    return any(os.path.getmtime(d) > t for d in [src, *deps])


BINDING_SRC = os.path.join(HERE, "python", "kvcache_b200", "csrc", "binding.cpp")
BINDING = os.path.join(HERE, "python", "kvcache_b200", "_binding.so")


def build_binding(force: bool = False) -> str:
    """The Python binding's native half (descriptors of torch tensors), against the installed torch."""
    import sysconfig

    import torch
    header = os.path.join(HERE, "..", "include", "kvcache_b200.h")
    tdir = os.path.dirname(torch.__file__)
    if force or _newer(BINDING_SRC, BINDING, [header, os.path.join(tdir, "version.py")]):
        inc = [sysconfig.get_paths()["include"], os.path.join(tdir, "include"),
               os.path.join(tdir, "include", "torch", "csrc", "api", "include"), "/usr/local/cuda/include"]
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
               *[f"-I{d}" for d in inc], BINDING_SRC, "-o", BINDING, f"-L{os.path.join(tdir, 'lib')}", "-ltorch_python",
               "-ltorch_cpu", "-lc10", "-lc10_cuda"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"g++ failed for the binding:\n{res.stdout}\n{res.stderr}")
    return BINDING


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(LIBDIR, exist_ok=True)
    nvcc = _nvcc()
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(HERE, "..", "include", "kvcache_b200.h"))
    sources = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]

    def compile_one(name: str):
        src = os.path.join(CSRC, name)
        obj = os.path.join(OBJ, name.replace(".cu", ".o"))
        if force or _newer(src, obj, headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
                print(" ".join(cmd))
            res = subprocess.run(cmd, capture_output=True, text=True)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed for {name}:\n{res.stdout}\n{res.stderr}")
            if verbose:
                print(res.stderr)
            return obj, True
        return obj, False

    with ThreadPoolExecutor(max_workers=min(8, len(sources))) as pool:
        binding = pool.submit(build_binding, force)
        results = list(pool.map(compile_one, sources))
        binding.result()
    objs = [o for o, _ in results]
    if force or any(changed for _, changed in results) or not os.path.exists(LIB):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-ldl", "-cudart", "static"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    args = ap.parse_args()
    print(build(force=args.force, verbose=args.verbose))
    sys.exit(0)
