"""Builds fp6_marlin_b200/libfp6m.so in-tree with nvcc for sm_100a (no GPU needed to compile).

Usage:  python fp6_marlin_b200/build.py [--force] [--verbose] [--trace]   (run as a script: it must
work before the package itself can be imported)
"""
from __future__ import annotations

import hashlib
import importlib.util
import os
import re
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libfp6m.so")
CALL_PATH = os.path.join(PKG_DIR, "_call.so")          # extension module: the Python call path of mul and mul_fused
CALL_SOURCES = [os.path.join(CSRC, "py_call.cpp"), os.path.join(os.path.dirname(PKG_DIR), "include", "fp6m.h")]
OBJ_DIR = os.path.join(PKG_DIR, "build")

CUDA_SOURCES = ["c_api.cu", "gemm_few.cu", "gemm_team.cu", "gemm_tc5.cu", "gemm_wide.cu", "dump_operands.cu", "prep_gpu.cu", "gather_columns.cu", "peer.cu"]
HOST_SOURCES = ["host_pack.cpp"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = os.path.join(cuda_home, "bin", "nvcc")
    return cand if os.path.isfile(cand) else (shutil.which("nvcc") or "nvcc")


def _sources() -> list[str]:
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(os.path.dirname(PKG_DIR), "include", "fp6m.h"))
    return [os.path.join(CSRC, f) for f in CUDA_SOURCES + HOST_SOURCES] + headers


def needs_build() -> bool:
    if not os.path.isfile(LIB_PATH):
        return True
    lib_time = os.path.getmtime(LIB_PATH)
    return any(os.path.getmtime(s) > lib_time for s in _sources())


def _torch_dir() -> str:
    """Where torch is installed (looked up, not imported)."""
    return importlib.util.find_spec("torch").submodule_search_locations[0]


def _call_command() -> list[str]:
    torch_dir = _torch_dir()
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    includes = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    with open(os.path.join(torch_dir, "version.py")) as f:
        version = re.search(r"^__version__ = '([^']+)'", f.read(), re.M).group(1)
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f'-DFP6M_TORCH_VERSION="{version}"', *[f"-isystem{i}" for i in includes],
            CALL_SOURCES[0], "-o", CALL_PATH, "-L" + os.path.join(torch_dir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]


def _call_stamp() -> str:
    """What the extension module depends on: its sources (the C ABI's declarations among them), the command, this Python, and torch,
    whose accessors it has inlined and whose fields it reads at their offsets."""
    digest = hashlib.sha256("\0".join([sys.version, *_call_command()]).encode())
    for path in [*CALL_SOURCES, os.path.join(_torch_dir(), "version.py")]:
        with open(path, "rb") as f:
            digest.update(f.read())
    return digest.hexdigest()


def build_call(force: bool = False) -> str:
    """Compile the extension module that reads torch tensors for mul and mul_fused (no CUDA code); returns its path."""
    stamp_path, stamp = os.path.join(OBJ_DIR, "_call.stamp"), _call_stamp()
    if not force and os.path.isfile(CALL_PATH) and os.path.isfile(stamp_path):
        with open(stamp_path) as f:
            if f.read() == stamp:
                return CALL_PATH
    os.makedirs(OBJ_DIR, exist_ok=True)
    subprocess.run(_call_command(), check=True)
    with open(stamp_path, "w") as f:
        f.write(stamp)
    return CALL_PATH


def build(force: bool = False, verbose: bool = False, trace: bool = False) -> str:
    """Compile every source to an object and link the shared library; returns its path.
    ``trace=True`` builds libfp6m_trace.so instead: the same library with the in-kernel timeline of
    csrc/trace.cuh compiled in (read by ``python -m fp6_marlin_b200.timeline``)."""
    if not trace:
        build_call(force)
    lib_path = os.path.join(PKG_DIR, "libfp6m_trace.so") if trace else LIB_PATH
    obj_dir = OBJ_DIR + ("_trace" if trace else "")
    if not force and not trace and not needs_build():
        return lib_path
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = _nvcc()
    objs, procs = [], []
    log = []
    for src in CUDA_SOURCES + HOST_SOURCES:
        obj = os.path.join(obj_dir, os.path.splitext(src)[0] + ".o")
        objs.append(obj)
        cmd = [nvcc, *NVCC_FLAGS, *(["-DFP6M_TRACE"] if trace else []), "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, proc in procs:
        out, _ = proc.communicate()
        log.append(f"==== {src}\n{out}")
        failed |= proc.returncode != 0
    text = "\n".join(log)
    with open(os.path.join(obj_dir, "ptxas.log"), "w") as f:
        f.write(text)
    if failed or verbose:
        print(text)
    if failed:
        raise RuntimeError("nvcc failed; see output above")
    subprocess.run([nvcc, "-shared", "-o", lib_path, *objs, "-lcudart"], check=True)
    return lib_path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, trace="--trace" in sys.argv))
