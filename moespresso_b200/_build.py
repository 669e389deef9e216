"""In-tree build of the CUDA extension: ``libmoespresso_b200.so`` next to this file, and ``_native.so``, the native host
calls over it.

Plain ``nvcc`` for sm_100a only; no torch headers are involved in the library because it is a C ABI (see
``include/moespresso_b200.h``).  ``_native.so`` is a CPython extension that knows torch tensors and holds no device code; it is
bound to one torch and one interpreter and has a stamp of its own that says which.
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
NATIVE_STAMP = os.path.join(HERE, "build", "native_stamp.txt")
HEADER = os.path.join(HERE, "..", "include", "moespresso_b200.h")
SOURCES = ["runtime.cu", "indexer_scores.cu", "indexer_scores_fp8.cu", "indexer_decode.cu", "indexer_qat.cu", "kv_formats.cu", "qwen_q8.cu", "topk_select.cu", "topk_multi.cu", "topk_pivot.cu", "sparse_attn.cu", "decode_fused.cu", "sparse_attn_tc.cu", "sparse_attn_few.cu", "flash_prefill.cu", "flash_single.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v",
]
GXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return exe


def _digest(paths, *more: str) -> str:
    h = hashlib.sha256()
    for path in paths:
        h.update(os.path.basename(path).encode())
        with open(path, "rb") as f:
            h.update(f.read())
    h.update(" ".join(more).encode())
    return h.hexdigest()


def _library_digest() -> str:
    device = [os.path.join(CSRC, n) for n in sorted(os.listdir(CSRC)) if n.endswith((".cu", ".cuh"))]
    return _digest([*device, HEADER], *NVCC_FLAGS)


def _native_digest() -> str:
    """What ``_native.so`` was compiled against besides its sources: torch's C++ classes and the interpreter."""
    import sysconfig

    import torch
    return _digest([os.path.join(CSRC, "host_calls.cpp"), HEADER], *GXX_FLAGS, torch.__version__, str(torch.version.git_version),
                   str(torch._C._GLIBCXX_USE_CXX11_ABI), str(sysconfig.get_config_var("SOABI")), sys.version)


def _stamped(built: str, stamp: str, digest) -> bool:
    if not (os.path.exists(built) and os.path.exists(stamp)):
        return False
    with open(stamp) as f:
        return f.read().strip() == digest()


def library_is_current() -> bool:
    return _stamped(LIB, STAMP, _library_digest)


def native_is_current() -> bool:
    return _stamped(NATIVE, NATIVE_STAMP, _native_digest)


def is_current() -> bool:
    return library_is_current() and native_is_current()


def _native_command(out: str):
    """g++ over torch's headers; the symbols come from the torch libraries that the process has loaded."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return ["g++", *GXX_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *(f"-I{d}" for d in inc), os.path.join(CSRC, "host_calls.cpp"), "-o", out, f"-L{os.path.join(root, 'lib')}",
            "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def _start(cmd):
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish(procs, log_name: str, verbose: bool) -> None:
    """Waits for (source, process) pairs, keeps their output; raises if one failed."""
    log = []
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        log.append(f"==== {src}\n{out}")
        failed |= pr.returncode != 0
    with open(os.path.join(HERE, "build", log_name), "w") as f:
        f.write("\n".join(log))
    if failed:
        sys.stderr.write("\n".join(log))
        raise RuntimeError(f"the build failed; see moespresso_b200/build/{log_name}")
    if verbose:
        print("\n".join(log))


def _write(stamp: str, digest: str) -> None:
    with open(stamp, "w") as f:
        f.write(digest)


def _native_part() -> str:
    """Where this process compiles to; moved into place when it is whole (another process may have the old one loaded)."""
    return os.path.join(HERE, "build", f"native.{os.getpid()}.part")


def _start_native():
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    return [("host_calls.cpp", _start(_native_command(_native_part())))]


def _finish_native(procs, verbose: bool) -> None:
    _finish(procs, "native.log", verbose)
    os.replace(_native_part(), NATIVE)
    _write(NATIVE_STAMP, _native_digest())


def build_native() -> str:
    """Compile the CPython extension; returns its path."""
    _finish_native(_start_native(), False)
    return NATIVE


def build_library(verbose: bool = False) -> str:
    """Compile every .cu file and link the shared library; returns its path."""
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        procs.append((src, _start([nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj])))
        objs.append(obj)
    _finish(procs, "nvcc.log", verbose)
    link = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart_static",
            "-Xcompiler", "-fPIC"]
    subprocess.run(link, check=True)
    _write(STAMP, _library_digest())
    return LIB


def build(force: bool = False, verbose: bool = False) -> str:
    """Build what is not current: the library and the CPython extension.  Returns the library's path."""
    native = _start_native() if force or not native_is_current() else []
    try:
        if force or not library_is_current():
            build_library(verbose)
    finally:
        if native:
            _finish_native(native, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
