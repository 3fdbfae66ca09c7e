"""Builds libsimplicial_attn_b200.so (the C-ABI library) in-tree with nvcc for sm_100a.

    python -m simplical_attn_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import concurrent.futures
import contextlib
import fcntl
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIB_DIR, "libsimplicial_attn_b200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared", "--expt-relaxed-constexpr", "-Xptxas", "-v",
]


def nvcc_path() -> str:
    return os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def have_compiler() -> bool:
    return os.path.exists(nvcc_path())


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


STAMP = LIB + ".sources"      # digest of the sources the library was built from


def _deps():
    deps = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC))
    deps.append(os.path.join(os.path.dirname(PKG), "include", "simplicial_attn_b200.h"))
    return deps


def source_digest() -> str:
    """Digest of every file the library is compiled from and of the compiler flags.  File times are not
    used: a copy of the tree (a checkout, an archive) need not preserve them."""
    h = hashlib.sha256(" ".join(NVCC_FLAGS).encode())
    for d in _deps():
        h.update(os.path.basename(d).encode())
        with open(d, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def _stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(STAMP):
        return True
    with open(STAMP) as f:
        return f.read().strip() != source_digest()


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library if it is missing or was built from other sources; returns its path.  Every
    .cu file of csrc/ is one translation unit; the units compile side by side and are then linked."""
    if not force and not _stale():
        return LIB
    nvcc = nvcc_path()
    os.makedirs(LIB_DIR, exist_ok=True)
    digest = source_digest()
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    compile_flags = [f for f in NVCC_FLAGS if f != "-shared"]

    def compile_one(src: str):
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        res = subprocess.run([nvcc] + compile_flags + ["-c", "-o", obj, src], capture_output=True, text=True)
        return obj, res

    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, min(len(sources()), os.cpu_count() or 1))) as pool:
        results = list(pool.map(compile_one, sources()))
    for _, res in results:
        if verbose or res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
    if any(res.returncode != 0 for _, res in results):
        raise RuntimeError("nvcc failed building " + LIB)
    link = subprocess.run([nvcc, "-shared", "-Xlinker", "-soname=" + os.path.basename(LIB), "-o", LIB] + [obj for obj, _ in results], capture_output=True, text=True)
    if verbose or link.returncode != 0:
        sys.stderr.write(link.stdout + link.stderr)
    if link.returncode != 0:
        raise RuntimeError("nvcc failed linking " + LIB)
    with open(STAMP, "w") as f:
        f.write(digest + "\n")
    return LIB


# ---- the torch binding: host code only, compiled by the C++ compiler against torch's headers
BINDING_SRC = os.path.join(PKG, "binding", "sa_torch.cpp")
BINDING = os.path.join(LIB_DIR, "sa_torch.so")
BINDING_STAMP = BINDING + ".sources"
CXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
CUDA_INCLUDE = os.path.join(os.path.dirname(os.path.dirname(nvcc_path())), "include")


def cxx_path() -> str:
    # the system compiler, not $CXX: one that links its own static libstdc++ breaks exceptions across torch's libraries
    return "g++"


def have_host_compiler() -> bool:
    return shutil.which(cxx_path()) is not None and os.path.exists(CUDA_INCLUDE)


def binding_digest() -> str:
    import torch
    h = hashlib.sha256(" ".join(CXX_FLAGS + [torch.__version__, sys.version]).encode())
    for d in (BINDING_SRC, os.path.join(os.path.dirname(PKG), "include", "simplicial_attn_b200.h")):
        with open(d, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def binding_stale() -> bool:
    """Whether the binding is missing or was built from other sources, for another torch or another Python."""
    if not os.path.exists(BINDING) or not os.path.exists(BINDING_STAMP):
        return True
    with open(BINDING_STAMP) as f:
        return f.read().strip() != binding_digest()


@contextlib.contextmanager
def _locked():
    os.makedirs(LIB_DIR, exist_ok=True)
    with open(os.path.join(LIB_DIR, ".lock"), "w") as f:
        fcntl.flock(f, fcntl.LOCK_EX)          # released when the file is closed
        yield


def build_binding(force: bool = False) -> str:
    """Compile the torch binding if it is stale.  One process builds, the others wait for it; the file and its stamp
    are put in place whole, so that a process that does not build never sees half of one."""
    if not force and not binding_stale():
        return BINDING
    with _locked():
        if force or binding_stale():
            _compile_binding()
    return BINDING


def _put(path: str, write) -> None:
    """Has `write` make a file beside `path`, then moves it there."""
    part = f"{path}.{os.getpid()}.part"
    try:
        write(part)
        os.replace(part, path)
    finally:
        if os.path.exists(part):
            os.remove(part)


def _write_text(text: str):
    def write(path):
        with open(path, "w") as f:
            f.write(text)
    return write


def _compile_binding() -> None:
    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), CUDA_INCLUDE,
           sysconfig.get_paths()["include"]]
    cmd = ([cxx_path()] + CXX_FLAGS + [f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + ["-I" + d for d in inc]
           + [BINDING_SRC, LIB, "-L" + os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
              "-ltorch_python", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"])

    def compile_to(path):
        res = subprocess.run(cmd + ["-o", path], capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("the C++ compiler failed building " + BINDING)

    digest = binding_digest()
    _put(BINDING, compile_to)
    _put(BINDING_STAMP, _write_text(digest + "\n"))


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_binding(force="--force" in sys.argv))
