"""Builds ``libxdk_b200.so`` (the C-ABI library) in-tree with nvcc for sm_100a, and ``_host.*.so`` (the native half of the
Python ops: checks, output allocation, launch) with the host compiler against the installed torch, if that is one with CUDA.

    python -m cross_dsl_kernels_b200.build        # rebuild if any source is newer

No GPU is needed to build: nvcc cross-compiles.  The CUDA runtime is linked
statically, so the library loads on a machine without a GPU (calls then return
an error status) and has no dependency on any Python package; only ``_host.*.so`` knows torch, whose version and
interpreter its name carries.  Without it the ops run all the same, checked in Python.
"""

from __future__ import annotations

import os
import pathlib
import shutil
import subprocess
import sys

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libxdk_b200.so"
SOURCES = ("abi.cu", "rmsnorm.cu", "gemv.cu", "gemv_tc.cu", "gemv_mma.cu", "rope_kv.cu", "w4a16.cu", "quantize.cu", "peer.cu", "swiglu.cu", "attention.cu", "unshard.cu")
ARCH_FLAGS = ("-gencode", "arch=compute_100a,code=sm_100a")


def _nvcc() -> str:
    found = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found (set CUDA_HOME)")
    return found


def host_target() -> pathlib.Path | None:
    """The native half to build for the running torch and interpreter; None where there is no torch with CUDA to link."""
    try:
        from torch.utils.cpp_extension import library_paths
    except ImportError:
        return None
    if not any((pathlib.Path(d) / "libc10_cuda.so").exists() for d in library_paths()):
        return None
    from ._native import host_path
    return host_path()


def needs_build() -> bool:
    built = [p for p in (LIB, host_target()) if p is not None]
    if not all(p.exists() for p in built):
        return True
    stamp = min(p.stat().st_mtime for p in built)
    deps = [CSRC / s for s in SOURCES] + list(CSRC.glob("*.cuh")) + [CSRC / "host.cpp", PKG.parent / "include" / "xdk_b200.h"]
    return any(d.stat().st_mtime > stamp for d in deps)


def _host_command(obj: pathlib.Path) -> list[str]:
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths

    cuda = pathlib.Path(_nvcc()).resolve().parent.parent / "include"
    dirs = [*include_paths(), str(cuda), sysconfig.get_paths()["include"]]
    abi = f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", abi, *(f"-I{d}" for d in dirs), "-c", str(CSRC / "host.cpp"),
            "-o", str(obj)]


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    """Compile every kernel translation unit and link the shared library."""
    if not force and not needs_build():
        return LIB
    nvcc = _nvcc()
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)
    common = [nvcc, *ARCH_FLAGS, "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    for src in SOURCES:
        obj = objdir / (src[:-3] + ".o")
        procs.append((src, subprocess.Popen(common + ["-c", str(CSRC / src), "-o", str(obj)],
                                            stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    host = host_target()
    if host is not None:
        procs.append(("host.cpp", subprocess.Popen(_host_command(objdir / "host.o"), stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                                   text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(f"--- {src}\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed; see output above")
    objs = [str(objdir / (s[:-3] + ".o")) for s in SOURCES]
    link = [nvcc, *ARCH_FLAGS, "-shared", "-cudart", "static", "-o", str(LIB), *objs]
    done = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if done.returncode:
        raise RuntimeError("link failed:\n" + done.stdout)
    if host is None:
        return LIB
    from torch.utils.cpp_extension import library_paths
    link = ["g++", "-shared", "-o", str(host), str(objdir / "host.o"), f"-L{PKG}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN",
            *(f"-L{d}" for d in library_paths()), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    cuda = pathlib.Path(nvcc).resolve().parent.parent / "lib64"
    done = subprocess.run(link + [f"-L{cuda}", "-lcudart"], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if done.returncode:
        raise RuntimeError("link failed:\n" + done.stdout)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
