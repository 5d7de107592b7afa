"""nvcc driver and in-tree cache for the core library and the generated modules.

Everything is compiled for sm_100a only and written under ``fasteq_b200/lib``
(git-ignored, shipped with the working tree).  Generated modules are keyed by a
hash of their operator signature plus the emitter version, the same role as the
reference's on-disk JIT cache (fasteq/ops/uniform1d_jit.py:444-471, :614-674),
without the auto-tuning sweep.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import threading
from typing import List, Optional

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIB = os.path.join(PKG, "lib")
JIT = os.path.join(LIB, "jit")
CORE_SO = os.path.join(LIB, "libfasteq_b200_core.so")
CORE_SOURCES = ["core.cu", "eqlinear.cu", "eqlinear_api.cu", "gemm_tf32x3.cu", "radial_chain.cu", "gate.cu", "neighbors.cu", "edge_geometry.cu", "silu.cu", "readout.cu"]

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-diag-suppress", "177",
          f"-I{INCLUDE}", f"-I{CSRC}"]
_lock = threading.Lock()


class BuildError(RuntimeError):
    pass


def nvcc_path() -> str:
    for cand in (os.environ.get("FASTEQ_NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise BuildError("nvcc not found: fasteq_b200 compiles its sm_100a kernels with nvcc and has no fallback path")


def compile_shared(sources: List[str], out_so: str, extra: Optional[List[str]] = None, verbose: bool = False) -> str:
    os.makedirs(os.path.dirname(out_so), exist_ok=True)
    tmp = out_so + f".tmp{os.getpid()}_{threading.get_ident()}"
    cmd = [nvcc_path()] + ARCH + COMMON + (extra or []) + ["-o", tmp] + sources
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise BuildError(f"nvcc failed ({' '.join(cmd)}):\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, out_so)
    if verbose:
        print(r.stdout, r.stderr)
    return r.stdout + r.stderr


def _newer(target: str, deps: List[str]) -> bool:
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(d) <= t for d in deps if os.path.exists(d))


def headers() -> List[str]:
    hs = [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    hs += [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    return hs


def build_core(force: bool = False) -> str:
    srcs = [os.path.join(CSRC, s) for s in CORE_SOURCES]
    with _lock:
        if force or not _newer(CORE_SO, srcs + headers()):
            compile_shared(srcs, CORE_SO, extra=["-Xptxas", "-v"])
    return CORE_SO


FRONT = os.path.join(CSRC, "front")
FRONT_SOURCES = ["module.cpp", "prepared.cpp", "layers.cpp", "edges.cpp", "u1d.cpp"]
_front_lock = threading.Lock()


def _loaded_runtime() -> List[str]:
    """The C++ runtime torch brought into this process.  The extension is linked to it by path: a compiler whose own is an archive would
    put a second one into the extension, and formatting a number with that one ends the process."""
    with open("/proc/self/maps") as f:
        return sorted({line.split()[-1] for line in f if os.path.basename(line.split()[-1]).startswith("libstdc++.so")})


def front_so() -> str:
    """Unlike the libraries behind the C interface the extension belongs to one torch, one interpreter and one ABI of the C++ runtime."""
    import sys
    import torch
    return os.path.join(LIB, f"fasteq_front.torch{torch.__version__}.abi{int(torch._C._GLIBCXX_USE_CXX11_ABI)}.{sys.implementation.cache_tag}.so")


def build_front(force: bool = False) -> str:
    """The native host path: host code only, compiled with g++ against torch's headers."""
    import sysconfig
    import tempfile
    from concurrent.futures import ThreadPoolExecutor
    so = front_so()
    srcs = [os.path.join(FRONT, s) for s in FRONT_SOURCES]
    deps = srcs + [os.path.join(FRONT, "front.h"), os.path.join(INCLUDE, "fasteq_b200.h")]
    with _front_lock:
        if not force and _newer(so, deps):
            return so
        import torch
        base = os.path.dirname(torch.__file__)
        cuda = os.path.dirname(os.path.dirname(nvcc_path()))
        cxx = os.environ.get("CXX") or shutil.which("g++")
        if not cxx:
            raise BuildError("g++ not found: fasteq_b200 compiles its host path with it and has no fallback path")
        flags = ["-O2", "-std=c++17", "-fPIC", "-DTORCH_EXTENSION_NAME=fasteq_front", "-DTORCH_API_INCLUDE_EXTENSION_H",
                 f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
        flags += [f"-I{p}" for p in (os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
                                     sysconfig.get_paths()["include"], os.path.join(cuda, "include"), INCLUDE)]
        os.makedirs(LIB, exist_ok=True)
        with tempfile.TemporaryDirectory(dir=LIB) as tmp:
            def run(cmd):
                r = subprocess.run(cmd, capture_output=True, text=True)
                if r.returncode != 0:
                    raise BuildError(f"{cmd[0]} failed ({' '.join(cmd)}):\n{r.stdout}\n{r.stderr}")
            objs = [os.path.join(tmp, s[:-4] + ".o") for s in FRONT_SOURCES]
            with ThreadPoolExecutor(len(srcs)) as ex:
                list(ex.map(lambda so: run([cxx] + flags + ["-c", so[0], "-o", so[1]]), zip(srcs, objs)))
            out = os.path.join(tmp, "fasteq_front.so")
            libs = os.path.join(base, "lib")
            run([cxx, "-shared", "-o", out] + objs + _loaded_runtime() + [f"-L{libs}", f"-Wl,-rpath,{libs}", f"-L{cuda}/lib64", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
                                                       "-ltorch_python", "-lc10", "-lc10_cuda", "-lcudart"])
            os.replace(out, so)
    return so


def build_generated(name: str, source: str, extra: Optional[List[str]] = None, force: bool = False) -> str:
    """Compile generated CUDA text into ``lib/jit/<name>.so`` unless an up-to-date build exists."""
    so = os.path.join(JIT, name + ".so")
    cu = os.path.join(JIT, name + ".cu")
    if not force and os.path.exists(so) and os.path.exists(cu):
        with open(cu) as f:
            if f.read() == source and _newer(so, headers()):
                return so
    os.makedirs(JIT, exist_ok=True)
    tmp_cu = cu + f".tmp{os.getpid()}_{threading.get_ident()}.cu"
    with open(tmp_cu, "w") as f:
        f.write(source)
    try:
        log = compile_shared([tmp_cu], so, extra=["-Xptxas", "-v"] + (extra or []))
    finally:
        if os.path.exists(tmp_cu):
            os.replace(tmp_cu, cu)
    with open(os.path.join(JIT, name + ".log"), "w") as f:
        f.write(log)
    return so
