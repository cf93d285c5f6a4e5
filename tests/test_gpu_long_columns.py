"""Columns of more warp windows (28 rows each) than a launch grid's y extent
holds, 65,535: they take further launches, and give the other kernels' bits."""
import numpy as np
import pytest

from hydro_b200 import Domain, make_params
from _helpers import bitwise_equal, describe_mismatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fma"])
@pytest.mark.parametrize("ny", [65535 * 28 - 2, 65535 * 28 + 30])
def test_windows_beyond_the_grid_s_y_extent(product_lib, precision, ny):
    H = make_params(3, ny)
    rng = np.random.default_rng(ny)
    u0 = np.empty((4, ny + 4, 7))
    u0[0] = 1.0 + 0.1 * rng.random(u0[0].shape)
    u0[1] = 0.1 * rng.random(u0[0].shape)
    u0[2] = 0.1 * rng.random(u0[0].shape)
    u0[3] = 2.5 + 0.1 * rng.random(u0[0].shape)
    out = []
    for k in ("warp", "coop"):
        d = Domain(H, precision=precision, kernels=(k, k))
        d.upload(u0)
        d.godunov(1, 1e-3, fuse_courant=True)
        out.append((d.download(), d.courant()))
        d.close()
    assert out[0][1] == out[1][1]
    assert bitwise_equal(out[0][0], out[1][0]), describe_mismatch(out[0][0], out[1][0])
