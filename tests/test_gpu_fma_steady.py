"""Steady cells of the FMA tier: a sweep leaves a cell's values as they are, exactly,
where the five cells around it along the line are alike, and its kernels give one
set of bits (the stages round the same way in each)."""
import numpy as np
import pytest

from hydro_b200 import Domain, make_params
from _helpers import bitwise_equal, describe_mismatch
from test_gpu_steady import SIZES, padded, patchwork, run

pytestmark = pytest.mark.gpu

KERNELS = [("march", "march"), ("warp", "warp"), ("coop", "coop"), ("coop8", "coop8")]


@pytest.mark.parametrize("n", range(len(SIZES)))
@pytest.mark.parametrize("kernels", KERNELS)
@pytest.mark.parametrize("idim", [1, 2])
def test_uniform_neighbourhoods_are_kept(product_lib, n, kernels, idim):
    nx, ny = SIZES[n]
    u0 = padded(patchwork(nx, ny, 11 * n + 1))
    d = Domain(make_params(nx, ny, boundary=(0, 0, 0, 0)), precision="fma", kernels=kernels)
    d.upload(u0)
    # The step's second sweep alone, behind one of no time, which may sign a zero.
    d.sweep(0, 3 - idim, 0.0)
    d.sweep(1, idim, 1e-4 / nx)
    got = d.download()
    d.close()
    inner = u0[:, 2:-2, 2:-2]
    axis = 2 if idim == 1 else 1
    alike = np.ones(inner.shape[1:], dtype=bool)
    n_in = u0.shape[axis] - 4
    for s in range(5):
        shifted = np.take(u0, range(s, s + n_in), axis)
        shifted = shifted[:, 2:-2] if idim == 1 else shifted[:, :, 2:-2]
        alike &= ((shifted == inner).all(0))
    assert alike.any()
    assert np.array_equal(got[:, 2:-2, 2:-2][:, alike], inner[:, alike])


@pytest.mark.parametrize("n", range(len(SIZES)))
def test_fma_kernels_give_one_set_of_bits(product_lib, n):
    nx, ny = SIZES[n]
    H = make_params(nx, ny)
    u0 = padded(patchwork(nx, ny, 11 * n + 1))
    want, clock = run(H, u0, "fma", ("march", "march"))
    for k in KERNELS[1:]:
        got, c = run(H, u0, "fma", k)
        assert c == clock
        assert bitwise_equal(got, want), describe_mismatch(got, want)
