"""Compile the CUDA sources under csrc/ into libq40b200.so (sm_100a only), in-tree.

    python -m spec_mcts_b200.build            # rebuild if a source is newer than the library
    python -m spec_mcts_b200.build --force

nvcc cross-compiles without a GPU, so this runs on a CPU-only machine too.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
BUILD = os.path.join(PKG_DIR, "build")
LIB = os.path.join(PKG_DIR, "libq40b200.so")
HOST_SRC = os.path.join(CSRC, "host_calls.cpp")          # Python extension: see there
HOST = os.path.join(PKG_DIR, "_host_calls" + sysconfig.get_config_var("EXT_SUFFIX"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


STAMP = LIB + ".sha"
HOST_STAMP = HOST + ".sha"


def _digest(files, *words: str) -> str:
    """Content hash of what something is built from (file times do not survive a copy of the tree to another machine,
    contents do)."""
    import hashlib
    h = hashlib.sha256(" ".join(words).encode())
    for f in files:
        h.update(os.path.basename(f).encode())
        h.update(open(f, "rb").read())
    return h.hexdigest()


def _sources_digest() -> str:
    return _digest(sources() + sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) +
                   sorted(glob.glob(os.path.join(PKG_DIR, "..", "include", "*.h"))), *NVCC_FLAGS)


def _host_digest() -> str:
    """... of the Python extension, which uses torch's C++ interface: that differs from version to version."""
    import torch
    return _digest([HOST_SRC], torch.__version__, str(torch.version.cuda), str(int(torch._C._GLIBCXX_USE_CXX11_ABI)))


def _is_built(path: str, stamp: str, digest: str) -> bool:
    return os.path.exists(path) and os.path.exists(stamp) and open(stamp).read().strip() == digest


def needs_build() -> bool:
    return not _is_built(LIB, STAMP, _sources_digest())


def host_needs_build() -> bool:
    return not _is_built(HOST, HOST_STAMP, _host_digest())


def build_host(force: bool = False) -> str:
    """Compile the Python extension, with the host's C++ compiler."""
    if not force and not host_needs_build():
        return HOST
    import torch
    t, new = os.path.dirname(torch.__file__), f"{HOST}.{os.getpid()}"
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I" + os.path.join(t, "include"),
           "-I" + os.path.join(t, "include", "torch", "csrc", "api", "include"), "-I" + sysconfig.get_paths()["include"],
           "-I" + os.path.join(cuda, "include"), HOST_SRC, "-o", new, "-L" + os.path.join(t, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"building {HOST_SRC} failed:\n{r.stdout}\n{r.stderr}")
    os.replace(new, HOST)              # a process that has the old one loaded keeps it
    with open(HOST_STAMP, "w") as f:
        f.write(_host_digest())
    return HOST


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    os.makedirs(BUILD, exist_ok=True)
    nvcc = _nvcc()
    flags = list(NVCC_FLAGS)
    objs = []

    def compile_one(src):
        obj = os.path.join(BUILD, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *flags, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(sources()) or 1)) as ex:
        objs = list(ex.map(compile_one, sources()))
    cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
           "-Xcompiler", "-fPIC"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    with open(STAMP, "w") as f:
        f.write(_sources_digest())
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
    print(build_host(force="--force" in sys.argv))
