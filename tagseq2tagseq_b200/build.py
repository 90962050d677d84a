"""Builds libts2ts_attn.so (hand-written sm_100a CUDA behind a C ABI) in-tree with nvcc.

    python -m tagseq2tagseq_b200.build [--force]

nvcc cross-compiles without a GPU.  The library links only the static CUDA runtime, so it
also loads on a machine without a driver (the symbol-export test does exactly that).
libts2ts_torch.so, plain C++ against the installed PyTorch, holds the torch operators that call it.

What a file was built from (sources, flags, the PyTorch version) is recorded beside the objects as a digest: a file is
rebuilt when its own record differs, whatever its age.  Files appear under their names only once they are complete, and
one process at a time builds.
"""
from __future__ import annotations

import contextlib
import fcntl
import hashlib
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(HERE, "..", "include")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libts2ts_attn.so")
SELFTEST_LIB = os.path.join(HERE, "libts2ts_selftest.so")  # test-only: the bounded-wait self-test kernel
TORCH_LIB = os.path.join(HERE, "libts2ts_torch.so")
SOURCES = ["api.cu", "block_map.cu", "link_scan.cu", "attn_fwd.cu", "attn_bwd.cu", "attn_decode.cu", "lm_fused.cu", "adamw.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--use_fast_math", "-Xptxas", "-v"]
IEEE_SOURCES = ("adamw.cu",)  # compiled without --use_fast_math
SELFTEST_FLAGS = [f for f in NVCC_FLAGS if f not in ("-Xptxas", "-v")] + ["-DTS2TS_SPIN_LIMIT=4096u"]


def _nvcc() -> str:
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return path


def _torch_flags() -> list:
    import torch
    root = os.path.dirname(torch.__file__)
    return ["-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", "-I/usr/local/cuda/include", os.path.join(CSRC, "torch_ops.cpp"),
            f"-L{HERE}", "-l:libts2ts_attn.so", f"-L{root}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-Wl,-rpath,$ORIGIN"]


# ------------------------------------------------------------------------------------------------ what a file is built from
def _headers() -> list:
    return [os.path.join(d, f) for d in (CSRC, INCLUDE) for f in sorted(os.listdir(d)) if f.endswith((".h", ".cuh"))]


def _digest(files, words) -> str:
    h = hashlib.sha256(repr(list(words)).encode())
    for f in files:
        with open(f, "rb") as fh:
            h.update(os.path.basename(f).encode() + b"\0" + fh.read() + b"\0")
    return h.hexdigest()


def _flags(src: str) -> list:
    return [f for f in NVCC_FLAGS if f != "--use_fast_math" or src not in IEEE_SOURCES]


def _object(src: str) -> str:
    return os.path.join(OBJ, src.replace(".cu", ".o"))


def _wanted(path: str) -> str:
    """Digest of everything the file at ``path`` is built from, as it stands now."""
    if path == TORCH_LIB:
        import torch
        return _digest([os.path.join(CSRC, "torch_ops.cpp"), *_headers()], ["torch", torch.__version__])
    if path == SELFTEST_LIB:
        return _digest([os.path.join(CSRC, "selftest_wait.cu"), *_headers()], SELFTEST_FLAGS)
    if path == LIB:
        return _digest([os.path.join(CSRC, s) for s in SOURCES] + _headers(), sum(map(_flags, SOURCES), []))
    src = next(s for s in SOURCES if _object(s) == path)
    return _digest([os.path.join(CSRC, src), *_headers()], _flags(src))


def _record(path: str) -> str:
    return os.path.join(OBJ, os.path.basename(path) + ".digest")


def _recorded(path: str):
    with contextlib.suppress(OSError):
        with open(_record(path)) as fh:
            return fh.read()
    return None


def unusable() -> list:
    """The libraries that cannot be loaded as they are: missing ones, and those known to be built from something else.  A
    library without a record (copied here by itself) is taken for what it says it is."""
    return [p for p in (LIB, TORCH_LIB) if not os.path.exists(p) or (_recorded(p) is not None and _recorded(p) != _wanted(p))]


def _up_to_date(path: str) -> bool:
    return os.path.exists(path) and _recorded(path) == _wanted(path)


# ------------------------------------------------------------------------------------------------ building
@contextlib.contextmanager
def _lock():
    os.makedirs(OBJ, exist_ok=True)
    with open(os.path.join(OBJ, ".lock"), "w") as fh:
        fcntl.flock(fh, fcntl.LOCK_EX)
        yield


def _make(path: str, command, what: str) -> str:
    """Run ``command(output)`` into a temporary file and put it in place of ``path`` with its record; returns the log."""
    digest, tmp = _wanted(path), f"{path}.{os.getpid()}.tmp"
    try:
        res = subprocess.run(command(tmp), capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"{what} failed to build:\n{res.stdout}\n{res.stderr}")
        with contextlib.suppress(FileNotFoundError):
            os.remove(_record(path))
        os.replace(tmp, path)
    finally:
        with contextlib.suppress(FileNotFoundError):
            os.remove(tmp)
    with open(_record(path), "w") as fh:
        fh.write(digest)
    return res.stderr


def build_library(force: bool = False, verbose: bool = False) -> str:
    with _lock():
        def compile_one(src):
            obj = _object(src)
            if not force and _up_to_date(obj):
                return ""
            return _make(obj, lambda out: [_nvcc(), *_flags(src), "-c", os.path.join(CSRC, src), "-o", out], src)

        if force or not _up_to_date(LIB):
            with ThreadPoolExecutor(max_workers=6) as ex:
                logs = list(ex.map(compile_one, SOURCES))
            if verbose:
                print("\n".join(logs))
            _make(LIB, lambda out: [_nvcc(), "-shared", "-o", out, *map(_object, SOURCES), "-cudart", "static"], "the kernel library")
        if force or not _up_to_date(SELFTEST_LIB):
            _make(SELFTEST_LIB, lambda out: [_nvcc(), *SELFTEST_FLAGS, "-shared", os.path.join(CSRC, "selftest_wait.cu"), "-o", out,
                                             "-cudart", "static"], "the self-test library")
        if force or not _up_to_date(TORCH_LIB):
            _make(TORCH_LIB, lambda out: [shutil.which("g++") or "g++", *_torch_flags(), "-o", out], "the torch operators")
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose=True))
