"""The bit-exact stages' quotients by a shared reciprocal (recip_rn, quot, quot1)
against the division, bit for bit: random operands, significands next to 1 and to
2, and numerators whose quotient lies next to the middle between two numbers (the
nearest to it that a numerator of 53 bits reaches)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hydro_b200",
                    "csrc")
SOURCE = r"""
#include "hb_stages.cuh"
__global__ void kernel(const double* a, const double* b, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const hb::Recip R = hb::make_recip(b[i]);
    out[i] = R.y;
    out[n + i] = hb::quot(a[i], R);
    out[2 * n + i] = hb::quot1(a[i], b[i], R.y);
}
extern "C" int quotients(const double* a, const double* b, double* out, int n) {
    double* d;
    if (cudaMalloc(&d, 5ull * n * 8)) return 1;
    cudaMemcpy(d, a, 8ull * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, 8ull * n, cudaMemcpyHostToDevice);
    kernel<<<(n + 255) / 256, 256>>>(d, d + n, d + 2ull * n, n);
    cudaMemcpy(out, d + 2ull * n, 24ull * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)cudaGetLastError();
}
"""


def operands():
    rng = np.random.default_rng(11)
    one, bits = 1 << 52, lambda n: [int(x) for x in rng.integers(1 << 52, 1 << 53, n)]
    near = list(range(one, one + 200)) + list(range(2 * one - 400, 2 * one - 1))
    near += [one + (1 << k) + j for k in range(52) for j in (-1, 0, 1) if one + (1 << k) + j >= one]
    a, b = [], []
    for B in near + bits(20000):
        for A in near[:8] + bits(4):
            a.append(A), b.append(B)
        # A 2^54 / B = Q - r / B with Q odd: A / B is a 54-bit number but for r.
        if B % 2:
            inverse = pow(B, -1, 1 << 54)
            for r in (-5, -3, -1, 1, 3, 5):
                Q = r * inverse % (1 << 54)
                A = (B * Q - r) >> 54
                if A >= one:
                    a.append(A), b.append(B)
    a, b = np.array(a, dtype=np.float64), np.array(b, dtype=np.float64)
    low = b.view(np.uint64) & np.uint64(0xffffffff)
    keep = low != 0xffffffff  # these are left to the division
    a, b = a[keep], b[keep]
    return (np.ldexp(a, rng.integers(-150, 50, a.size)) * rng.choice([-1.0, 1.0], a.size),
            np.ldexp(b, rng.integers(-150, 50, b.size)))


def test_quotients_equal_the_division(tmp_path):
    if not shutil.which("nvcc"):
        pytest.skip("built with nvcc")
    src, so = str(tmp_path / "q.cu"), str(tmp_path / "q.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "--fmad=false", "-Xcompiler", "-fPIC", "-shared", f"-I{CSRC}", "-o", so, src],
                   check=True)
    a, b = operands()
    assert a.size > 200000
    out = np.zeros((3, a.size))
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))
    assert C.CDLL(so).quotients(p(a), p(b), p(out), C.c_int(a.size)) == 0
    for got, want in zip(out, (1.0 / b, a / b, a / b)):
        assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
