"""Builds liblight_b200.so in-tree with nvcc for sm_100a (the only target), and _host.so, the native host path in
front of its hot entry points (csrc/host.cpp), against the installed torch."""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "liblight_b200.so")
HOST = os.path.join(HERE, "_host.so")
SOURCES = ["abi.cu", "gguf_dequant.cu", "gguf_matmul_generic.cu", "gguf_gemv_fast.cu", "gguf_gemv_batch.cu", "prefill_umma.cu", "decode_umma.cu", "int4.cu", "fp8_block.cu",
           "moe.cu", "peer_gather.cu", "decode_attn.cu", "norm_rope.cu", "w8a8.cu", "moe_route.cu", "decode_chain.cu", "gemv_bf16.cu", "moe_elementwise.cu", "router.cu", "gguf_decode_nt.cu", "gguf_decode_ts.cu",
           "gemm_tmem.cu", "decode_tmem.cu"]
NVCC_FLAGS = os.environ.get("LIGHT_B200_NVCC_EXTRA", "").split() + ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "-Xcompiler", "-fvisibility=hidden", "-Xptxas", "-v"]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: liblight_b200.so cannot be built on this machine")
    return nvcc


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles every .cu under csrc/ to an object and links the shared library.  Returns its path."""
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "light_b200.h"))
    objs = [os.path.join(objdir, src.replace(".cu", ".o")) for src in SOURCES]

    def compile_one(src_obj):
        s, o = os.path.join(CSRC, src_obj[0]), src_obj[1]
        if force or _stale(o, [s] + headers):
            return src_obj, subprocess.run([nvcc, *NVCC_FLAGS, "-c", s, "-o", o], capture_output=True, text=True)
        return src_obj, None

    with concurrent.futures.ThreadPoolExecutor(os.cpu_count() or 1) as pool:
        for (src, o), r in pool.map(compile_one, zip(SOURCES, objs)):
            if r is None:
                continue
            if verbose or r.returncode:
                sys.stderr.write(r.stdout + r.stderr)
            if r.returncode:
                raise RuntimeError(f"nvcc failed on {src}")
            with open(o + ".ptxas.txt", "w") as f:
                f.write(r.stderr)
    if force or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link of liblight_b200.so failed")
    build_host(force)
    return LIB


def build_host(force: bool = False) -> str:
    """Compiles csrc/host.cpp as the extension module light_b200._host, linked to liblight_b200.so beside it."""
    import sysconfig

    import torch

    src = os.path.join(CSRC, "host.cpp")
    if not (force or _stale(HOST, [src, os.path.join(HERE, "..", "include", "light_b200.h")])):
        return HOST
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"), "-isystem", cuda, "-isystem", sysconfig.get_paths()["include"],
           src, "-o", HOST, "-L" + libs, "-L" + HERE, "-l:liblight_b200.so", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed on host.cpp")
    return HOST


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
