"""Domains before and after the program resets the device (cudaDeviceReset ends
the program's own context): in a process of its own, through another copy of the
CUDA runtime than the library's, as an application has one."""
import glob
import os
import site
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes, sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
from hydro_b200 import Domain, make_params
from _helpers import random_state
runtime = ctypes.CDLL(sys.argv[2])
H = make_params(50, 40)
u0 = random_state(50, 40, 1, "smooth")

def maxima():
    d = Domain(H)
    d.upload(u0)
    d.godunov(2, 1e-6, fuse_courant=True)
    got = d.courant()
    d.close()
    return got

first = maxima()
for _ in range(2):
    assert runtime.cudaDeviceReset() == 0
    assert maxima() == first and first[0] > 1.0
"""


def test_domains_after_a_reset(product_lib):
    where = [os.path.join(p, "nvidia/cuda_runtime/lib") for p in site.getsitepackages()]
    found = [f for p in where + ["/usr/local/cuda/lib64"]
             for f in glob.glob(os.path.join(p, "libcudart.so.1*"))]
    if not found:
        pytest.skip("no shared CUDA runtime library")
    subprocess.run([sys.executable, "-c", PROGRAM, ROOT, found[0]], check=True, timeout=120)
