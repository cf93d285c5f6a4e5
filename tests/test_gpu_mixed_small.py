"""Small mixed grids take one cell per lane in both directions (28 outputs a
window): at the windows' edges and on both sides of the size where the two-cell
windows and the marcher begin, the results are the cooperative windows' bits."""
import numpy as np
import pytest

from hydro_b200 import Domain, make_params
from _helpers import bitwise_equal, describe_mismatch, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3, 3), (25, 27), (26, 28), (27, 29), (54, 55), (57, 83),
                                   (250, 125), (512, 512), (513, 512), (64, 4096), (4097, 64)])
@pytest.mark.parametrize("bnd", [(1, 1, 1, 1), (3, 3, 2, 1)])
def test_one_cell_windows_equal_the_cooperative_ones(product_lib, nx, ny, bnd):
    H = make_params(nx, ny, boundary=bnd, scheme=1 + nx % 3)
    u0 = random_state(nx, ny, nx + ny, "smooth")
    out = []
    for k in ((None, None), ("coop", "coop")):
        d = Domain(H, precision="mixed", kernels=k)
        d.upload(u0)
        d.set_clock()
        d.launch_steps(5)
        out.append((d.download(), d.get_clock()))
        d.close()
    assert np.isfinite(out[0][0]).all()
    assert out[0][1] == out[1][1]
    assert bitwise_equal(out[0][0], out[1][0]), describe_mismatch(out[0][0], out[1][0])
