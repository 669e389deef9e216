"""In-tree build of the CUDA extension: ``libmoespresso_b200.so`` next to this file, and ``_native.so``, the native host
calls over it.

Plain ``nvcc`` for sm_100a only; no torch headers are involved in the library because it is a C ABI (see
``include/moespresso_b200.h``).  ``_native.so`` is a CPython extension that knows torch tensors and holds no device code.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmoespresso_b200.so")
NATIVE = os.path.join(HERE, "_native.so")
STAMP = os.path.join(HERE, "build", "stamp.txt")
SOURCES = ["runtime.cu", "indexer_scores.cu", "indexer_scores_fp8.cu", "indexer_decode.cu", "indexer_qat.cu", "kv_formats.cu", "qwen_q8.cu", "topk_select.cu", "topk_multi.cu", "topk_pivot.cu", "sparse_attn.cu", "decode_fused.cu", "sparse_attn_tc.cu", "sparse_attn_few.cu", "flash_prefill.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return exe


def _digest() -> str:
    h = hashlib.sha256()
    names = sorted(os.listdir(CSRC)) + ["../../include/moespresso_b200.h"]
    for n in names:
        path = os.path.join(CSRC, n)
        if os.path.isfile(path):
            h.update(n.encode())
            with open(path, "rb") as f:
                h.update(f.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def is_current() -> bool:
    if not (os.path.exists(LIB) and os.path.exists(NATIVE) and os.path.exists(STAMP)):
        return False
    with open(STAMP) as f:
        return f.read().strip() == _digest()


def _native_command():
    """g++ over torch's headers; the symbols come from the torch libraries that the process has loaded."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *(f"-I{d}" for d in inc), os.path.join(CSRC, "host_calls.cpp"), "-o", NATIVE, f"-L{os.path.join(root, 'lib')}",
            "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu file and link the shared library; returns its path."""
    if not force and is_current():
        return LIB
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    procs.append(("host_calls.cpp", subprocess.Popen(_native_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    log = []
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        log.append(f"==== {src}\n{out}")
        failed |= pr.returncode != 0
    with open(os.path.join(HERE, "build", "nvcc.log"), "w") as f:
        f.write("\n".join(log))
    if failed:
        sys.stderr.write("\n".join(log))
        raise RuntimeError("the build failed; see moespresso_b200/build/nvcc.log")
    if verbose:
        print("\n".join(log))
    link = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart_static",
            "-Xcompiler", "-fPIC"]
    subprocess.run(link, check=True)
    with open(STAMP, "w") as f:
        f.write(_digest())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
