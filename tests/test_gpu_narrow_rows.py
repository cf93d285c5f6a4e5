"""Rows of at most half as many warp windows (28 outputs each) as a CTA has warps:
the CTA's warps take several rows once there are more rows than the GPU holds
CTAs.  At the windows' edges and with rows left over, whole and in the parts of a
split sweep, the results are the cooperative windows' bits."""
import numpy as np
import pytest

from hydro_b200 import Domain, make_params
from _helpers import bitwise_equal, describe_mismatch, random_state

pytestmark = pytest.mark.gpu

# One to five windows of 28 a row: 26, 54, 82, 110, 138 cells at most; then nine.
WIDTHS = [3, 26, 27, 54, 55, 82, 83, 110, 111, 138, 250]


@pytest.mark.parametrize("precision", ["fp64", "fma"])
@pytest.mark.parametrize("parts", [False, True])
@pytest.mark.parametrize("ny", [50, 592, 593, 1187, 2405])
@pytest.mark.parametrize("nx", WIDTHS)
def test_narrow_rows_equal_the_cooperative_windows(product_lib, precision, parts, nx, ny):
    H = make_params(nx, ny, boundary=(3, 3, 2, 1), scheme=1 + nx % 3,
                    slope_type=1.5 if nx % 2 else 1.0)
    u0 = random_state(nx, ny, nx + ny, "smooth")
    out = []
    for k in ("warp", "coop"):
        d = Domain(H, precision=precision, kernels=(k, k))
        d.upload(u0)
        for idim in (1, 2):
            for stage in (0, 1):
                for part in ((1, 2) if parts and k == "warp" else (0,)):
                    d.sweep(stage, idim if stage == 0 else 3 - idim, 1e-4 / nx,
                            fuse_courant=stage == 1, part=part)
        out.append((d.download(), d.courant()))
        d.close()
    assert np.isfinite(out[0][0]).all()
    assert out[0][1] == out[1][1]
    assert bitwise_equal(out[0][0], out[1][0]), describe_mismatch(out[0][0], out[1][0])
