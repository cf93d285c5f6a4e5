"""Mixed kernels on grids above the small ones, where the default takes two
cells a lane along x (one window a warp, or pipelined runs of windows copied by
cp.async once there are enough rows) and marches along y: on patchworks of
uniform states, with odd and even row pitch, all kernels give one set of bits."""
import numpy as np
import pytest

from hydro_b200 import make_params
from _helpers import bitwise_equal, describe_mismatch
from test_gpu_steady import padded, patchwork, run

pytestmark = pytest.mark.gpu


# 700 rows: one window a warp.  4800 rows of two runs each: pipelined.
@pytest.mark.parametrize("nx,ny", [(501, 700), (502, 700), (361, 4800), (362, 4800)])
@pytest.mark.parametrize("bnd", [(1, 1, 1, 1), (3, 3, 2, 1)])
def test_two_cell_windows_equal_the_marches(product_lib, nx, ny, bnd):
    H = make_params(nx, ny, boundary=bnd)
    u0 = padded(patchwork(nx, ny, nx + ny, patches=60))
    want, clock = run(H, u0, "mixed", ("march", "march"))
    assert np.isfinite(want).all()
    for k in [(None, None), ("warp", None), ("bulk", None), ("coop", "coop")]:
        got, c = run(H, u0, "mixed", k)
        assert c == clock
        assert bitwise_equal(got, want), describe_mismatch(got, want)
