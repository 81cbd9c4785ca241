"""Builds csrc/*.cu into the in-tree C-ABI shared libraries with nvcc for sm_100a only.

`python text-generation-inference_b200/build.py [--force] [--verbose] [--seq]`
  libb200_tgis.so  every source: the whole C ABI of include/b200_tgis.h
  libb200_seq.so   the sources the hybrid decoder families need (seq_*.cu + the block allocator and the runtime pieces); a
                   process that serves only such a model builds and loads this one (`--seq`, `build(target="seq")`)
  _b200_host.so    csrc/host/host_calls.cpp: the operators' per-call host work as a CPython extension over torch's C++ headers.  It saves time only:
                   where it cannot be built (no headers of Python's or torch's) or is another Python's or torch's, the same calls go through Python
Objects are shared between the first two.  The libraries are git-ignored; they are built in the tree at first use.
"""
from __future__ import annotations

import concurrent.futures
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(HERE, "libb200_tgis.so")
SEQ_LIB = os.path.join(HERE, "libb200_seq.so")
HOST_SRC = os.path.join(CSRC, "host", "host_calls.cpp")
HOST_LIB = os.path.join(HERE, "_b200_host.so")
SEQ_EXTRA_SOURCES = ("runtime.cu", "kv_alloc.cu", "gemm_f16.cu")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v",
]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: the B200 path cannot be built (there is no CPU fallback)")
    return nvcc


def sources(target: str = "all"):
    every = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    if target == "seq":
        return [f for f in every if f.startswith("seq_") or f in SEQ_EXTRA_SOURCES]
    return every


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def host_tag() -> str:
    """what a built _b200_host.so names itself: it fits one Python and one torch only"""
    return "b200_host for python %d.%d, torch %s;" % (*sys.version_info[:2], importlib.metadata.version("torch"))


def host_fits() -> bool:
    try:
        with open(HOST_LIB, "rb") as f:
            return host_tag().encode() in f.read()
    except (OSError, importlib.metadata.PackageNotFoundError):
        return False


def build_host(force: bool = False) -> None:
    if not force and not _stale(HOST_LIB, [HOST_SRC]) and host_fits():
        return
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    part = f"{HOST_LIB}.{os.getpid()}.part"
    includes = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
                os.path.join(cuda, "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-D_GLIBCXX_USE_CXX11_ABI=1", f'-DB200_HOST_TAG="{host_tag()}"', *(f"-I{d}" for d in includes), HOST_SRC,
           "-o", part, f"-L{os.path.join(torch_dir, 'lib')}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed on host_calls.cpp")
    os.replace(part, HOST_LIB)


def build(force: bool = False, verbose: bool = False, target: str = "all") -> str:
    """target "all": both libraries; "seq": libb200_seq.so only (compiles nothing else)."""
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "b200_tgis.h"))
    headers = [h for h in headers if os.path.exists(h)]
    jobs = []
    for src in sources(target):
        obj = os.path.join(OBJ, src[:-3] + ".o")
        if force or _stale(obj, [os.path.join(CSRC, src)] + headers):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-I", os.path.join(os.path.dirname(HERE), "include"), "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, 1 + len(jobs))) as ex:
        host = ex.submit(build_host, force)
        for src, r in ex.map(compile_one, jobs):
            if r.returncode != 0:
                sys.stderr.write(r.stdout + r.stderr)
                raise RuntimeError(f"nvcc failed on {src}")
            if verbose:
                sys.stderr.write(f"== {src}\n{r.stderr}\n")
            with open(os.path.join(OBJ, src[:-3] + ".ptxas.txt"), "w") as f:
                f.write(r.stderr)
        try:
            host.result()
        except Exception as e:
            sys.stderr.write(f"{HOST_LIB} could not be built ({e}): calls go through Python\n")
    for lib, which in ((LIB, "all"), (SEQ_LIB, "seq")):
        if target == "seq" and which == "all":
            continue
        objs = [os.path.join(OBJ, s[:-3] + ".o") for s in sources(which)]
        if force or _stale(lib, objs):
            part = f"{lib}.{os.getpid()}.part"  # linked aside and renamed: a concurrent first use never loads half a file
            cmd = [nvcc, "-shared", "-o", part, *objs, "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a"]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                sys.stderr.write(r.stdout + r.stderr)
                raise RuntimeError("link failed")
            os.replace(part, lib)
    return SEQ_LIB if target == "seq" else LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, target="seq" if "--seq" in sys.argv else "all"))
