"""The library's host code on a stand-in for the CUDA runtime (fake_cudart.cpp,
fake_kernels.cu): its object files linked with the stand-in, in place of the
CUDA runtime library.  Memory is host memory and kernels are recorded, not run."""
import ctypes as C
import os
import re
import shutil
import subprocess

import pytest

from hydro_b200 import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "hydro_b200", "csrc")


def build(outdir):
    if not shutil.which("nvcc") or not shutil.which("g++"):
        pytest.skip("the stand-in runtime is built with nvcc and g++")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc"))))
    run = lambda *a: subprocess.run(a, check=True, cwd=HERE)
    run("make", "-s", "-C", CSRC)
    so, a, b = (os.path.join(outdir, n) for n in ("libfake.so", "a.o", "b.o"))
    run("g++", "-std=c++17", "-O1", "-fPIC", f"-I{cuda}/include", "-c", "-o", a, "fake_cudart.cpp")
    run("nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
        f"-I{CSRC}", "-c", "-o", b, "fake_kernels.cu")
    objs = sorted(os.path.join(CSRC, "_build", f) for f in os.listdir(os.path.join(CSRC, "_build"))
                  if f.endswith(".o"))
    run("g++", "-shared", "-Wl,-Bsymbolic", "-o", so, a, b, *objs, "-lpthread")
    lib = C.CDLL(so)
    for name, res, args in _lib.SIGNATURES:
        f = getattr(lib, name)
        f.restype, f.argtypes = res, args
    lib.fake_launched.restype = lib.fake_faults.restype = C.c_char_p
    lib.fake_refuse.argtypes = [C.c_char_p]
    return lib


def launched(lib):
    """[(kernel, (grid x, y, z))] since the last call, kernels by their plain names."""
    out = []
    for rec in lib.fake_launched().decode().split(";")[:-1]:
        name, *g = rec.split()
        m = re.match(r"_ZN2hb(\d+)", name)  # the mangled hb::<name of that length>
        out.append((name[m.end():][:int(m.group(1))] if m else name, tuple(map(int, g))))
    return out
