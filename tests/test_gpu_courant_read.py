"""The Courant maxima reduced inside a step's second sweep, read by the host:
they are the standalone reduction's over the same state, a second read gives
them again, and nothing of an earlier, faster state is left in them, whether
the step is launched or replayed from a captured graph."""
import numpy as np
import pytest
import torch

from hydro_b200 import Domain, make_params

pytestmark = pytest.mark.gpu


def state(H, speed, seed):
    rng = np.random.default_rng(seed)
    u = np.zeros((4, H.ny + 4, H.nx + 4))
    n = (H.ny, H.nx)
    c = (slice(2, -2), slice(2, -2))
    u[0][c] = 1.0 + 0.1 * rng.random(n)
    u[1][c] = speed * (rng.random(n) - 0.5)
    u[2][c] = speed * (rng.random(n) - 0.5)
    u[3][c] = 1.0 + (u[1][c] ** 2 + u[2][c] ** 2) / u[0][c]
    return u


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("kernel", ["auto", "march", "coop"])
@pytest.mark.parametrize("precision", ["fp64", "fma", "mixed"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (250, 125)])
def test_fused_maxima_are_the_state_s_own(nx, ny, precision, kernel, captured):
    H = make_params(nx, ny)
    d = Domain(H, precision=precision, kernels=(kernel, kernel))
    stream = torch.cuda.ExternalStream(d.stream_ptr)
    d.upload(state(H, 50.0, 1))
    d.godunov(1, 1e-6, fuse_courant=True)
    fast = d.courant()
    d.upload(state(H, 0.5, 2))
    if captured:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            d.godunov(2, 1e-6, fuse_courant=True)
        with torch.cuda.stream(stream):
            g.replay()
    else:
        d.godunov(2, 1e-6, fuse_courant=True)
    first, again = d.courant(), d.courant()
    fresh = Domain(H, precision=precision)
    fresh.upload(d.download())
    assert first == again == fresh.courant()
    assert first[0] < fast[0] and first[1] < fast[1]


def test_more_domains_than_pairs_of_host_memory():
    """The mapped host memory the maxima are written to holds 256 pairs; domains
    beyond that read their slots by a copy."""
    H = make_params(3, 3)
    u = state(H, 0.5, 3)
    doms = [Domain(H) for _ in range(258)]
    for d in doms:
        d.upload(u)
    got = {d.courant() for d in doms}
    assert len(got) == 1
    for d in doms:
        d.close()
    d = Domain(H)
    d.upload(u)
    assert {d.courant()} == got
