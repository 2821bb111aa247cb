"""Builds the engine's shared library, ``pfsoftlib_b200/libpfsoft_b200.so``, with nvcc for
sm_100a only. Run ``python -m pfsoftlib_b200.build`` or call ``build()``.

The library is plain C ABI (include/pfsoft_b200.h); Python reaches it through ctypes and C/C++
callers link it directly. It is built in-tree so that it ships with the package directory.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB = os.path.join(HERE, "libpfsoft_b200.so")
CSRC = os.path.join(HERE, "csrc")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
              "-Xptxas", "-warn-spills"]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def host_compiler() -> list[str]:
    # the image's default $CXX wrapper is incomplete; the system g++ is the supported host compiler
    gxx = "/usr/bin/g++"
    return ["-ccbin", gxx] if os.path.exists(gxx) else []


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))


# sources compiled several times, once for each part that they define (a module of its own each)
PARTS = {"dwt_fixed.cu": ("DWT_PART", 13),   # kFixedParts in dwt.cuh
         "fft_two_kind.cu": ("FFT_KIND", 7)}   # kKinds in fft_two.cuh


def units() -> list[tuple[str, str, list[str]]]:
    """(source, object name, extra flags) of every compilation."""
    out = []
    for src in sources():
        name = os.path.basename(src)
        macro, n = PARTS.get(name, ("", 1))
        out += [(src, f"{name}.{i}.o" if macro else f"{name}.o", [f"-D{macro}={i}"] if macro else []) for i in range(n)]
    return out


def up_to_date() -> bool:
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(CSRC, "*.hpp")) + \
        glob.glob(os.path.join(ROOT, "include", "*.h"))
    return all(os.path.getmtime(d) <= t for d in deps)


def build(force: bool = False, verbose: bool = False, extra: list[str] | None = None) -> str:
    if not force and up_to_date():
        return LIB
    objdir = os.path.join(HERE, "_build")
    os.makedirs(objdir, exist_ok=True)
    objs = []
    procs = []
    for src, name, flags in units():
        obj = os.path.join(objdir, name)
        cmd = [nvcc(), *host_compiler(), *ARCH, *NVCC_FLAGS, *flags, *(extra or []), "-I", os.path.join(ROOT, "include"),
               "-c", src, "-o", obj]
        if verbose:
            print(" ".join(cmd))
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if out.strip():
            sys.stderr.write(out)
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"nvcc failed on {src}\n")
    if failed:
        raise RuntimeError("CUDA build failed")
    tmp = LIB + ".tmp"
    link = [nvcc(), *host_compiler(), *ARCH, "-shared", "-o", tmp, *objs, "-lcudart"]
    if verbose:
        print(" ".join(link))
    subprocess.run(link, check=True)
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
