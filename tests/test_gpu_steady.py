"""Steady cells: sweeps store u + 0 where five neighbours along the line hold
the same bits (zeros of either sign in the normal momentum count as one), and
the cooperative sweeps hand only the other windows to the second launch.
Patchworks of uniform rectangles put every edge of a uniform region at every
place of a window, with gas at rest, moving gas and signed zeros, beside each
kind of wall."""
import numpy as np
import pytest

from hydro_b200 import Domain, make_params
from _helpers import bitwise_equal, describe_mismatch, orc_from_H

pytestmark = pytest.mark.gpu


def patchwork(nx, ny, seed, patches=14):
    """Uniform background at rest with rectangles of other uniform states;
    ghost cells hold zeros, as the reference starts."""
    rng = np.random.default_rng(seed)
    u = np.zeros((4, ny + 4, nx + 4))
    zero = np.array([0.0, -0.0])
    u[0, 2:-2, 2:-2] = 1.0
    u[1, 2:-2, 2:-2] = zero[seed % 2]
    u[3, 2:-2, 2:-2] = 1e-5 if seed % 3 else 2.5
    for k in range(patches):
        i0, j0 = rng.integers(2, nx + 2), rng.integers(2, ny + 2)
        i1, j1 = min(nx + 2, i0 + rng.integers(1, nx)), min(ny + 2, j0 + rng.integers(1, ny))
        r, p = rng.choice([1.0, 0.5, 2.0]), rng.choice([1.0, 1e-3])
        mx, my = rng.choice([0.0, -0.0, 0.3, -0.2], 2)
        # A third of the patches differ from what they cover in one place only.
        if k % 3 == 0:
            u[k % 4, j0, i0] *= 1.0 + 1e-12
            continue
        box = (slice(j0, j1), slice(i0, i1))
        u[0][box], u[1][box], u[2][box] = r, mx, my
        u[3][box] = p / 0.4 + 0.5 * (mx * mx + my * my) / r
    return u


SIZES = [(61, 47), (130, 67), (128, 252), (251, 129), (64, 64), (3, 190), (190, 3)]
WALLS = [(1, 1, 1, 1), (2, 2, 2, 2), (3, 3, 3, 3), (0, 2, 1, 0)]


@pytest.mark.parametrize("n", range(len(SIZES)))
@pytest.mark.parametrize("bnd", WALLS)
@pytest.mark.parametrize("kernels", [("warp", "warp"), ("coop", "coop"), ("coop8", "coop8"),
                                     ("march", "march")])
def test_patchworks_match_oracle(product_lib, oracle, n, bnd, kernels):
    nx, ny = SIZES[n]
    H = make_params(nx, ny, boundary=bnd, scheme=1 + n % 3)
    u0 = patchwork(nx, ny, 7 * n + len(kernels[0]))
    p = orc_from_H(oracle, H)
    want = u0.copy()
    steps, dts, t = oracle.run(p, want, 7)
    d = Domain(H, kernels=kernels)
    d.upload(u0)
    d.set_clock()
    d.launch_steps(7)
    got = d.download()
    tg, ng, dt = d.get_clock()
    cx, cy = d.courant()
    d.close()
    assert ng == steps == 7 and dt == dts[-1] and tg == t
    assert bitwise_equal(got, want), describe_mismatch(got, want)
    _, ox, oy = oracle.courant(p, want)
    assert (cx, cy) == (ox, oy)


def padded(u):
    """Ghosts as the cells inside them (the FP32 stages need theirs in range)."""
    u[:, :, :2], u[:, :, -2:] = u[:, :, 2:3], u[:, :, -3:-2]
    u[:, :2], u[:, -2:] = u[:, 2:3], u[:, -3:-2]
    return u


def run(H, u0, precision, kernels):
    d = Domain(H, precision=precision, kernels=kernels)
    d.upload(u0)
    d.set_clock()
    d.launch_steps(7)
    out = d.download(), d.get_clock()
    d.close()
    return out


@pytest.mark.parametrize("n", range(len(SIZES)))
@pytest.mark.parametrize("bnd", WALLS)
def test_mixed_kernels_that_look_equal_those_that_do_not(product_lib, n, bnd):
    """The mixed marches have no steady path: the other kernels give their bits."""
    nx, ny = SIZES[n]
    H = make_params(nx, ny, boundary=bnd)
    u0 = padded(patchwork(nx, ny, 11 * n + 1))
    want, clock = run(H, u0, "mixed", ("march", "march"))
    assert np.isfinite(want).all()
    for k in [("warp", None), ("bulk", None), ("coop", "coop"), ("coop8", "coop8")]:
        got, c = run(H, u0, "mixed", k)
        assert c == clock
        assert bitwise_equal(got, want), describe_mismatch(got, want)


@pytest.mark.parametrize("n", range(len(SIZES)))
@pytest.mark.parametrize("kernels", [("march", "march"), ("warp", "warp"), ("coop", "coop")])
def test_fma_patchworks_against_the_oracle(product_lib, oracle, n, kernels):
    """The FMA tier's bound (1e-12 of the field's largest value; its general
    update may keep the rounding of a product that a steady cell's drops)."""
    nx, ny = SIZES[n]
    H = make_params(nx, ny)
    u0 = padded(patchwork(nx, ny, 11 * n + 1))
    want = u0.copy()
    oracle.run(orc_from_H(oracle, H), want, 7)
    got, _ = run(H, u0, "fma", kernels)
    for v in range(4):
        assert np.abs(got[v] - want[v]).max() <= 1e-12 * np.abs(want[v]).max()
