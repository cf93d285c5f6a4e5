"""The bit-exact FP64 stages where their shortcuts end: quotients of a shared
reciprocal hold within an exponent range and away from significands of ones,
the Newton step and the wave selection are compared instead of formed unless
the comparison is too near.  States beyond each of these limits, every cell
and the dt bit for bit against the oracle."""
import numpy as np
import pytest

from hydro_b200 import Domain, make_params
from _helpers import bitwise_equal, describe_mismatch, orc_from_H, random_state

pytestmark = pytest.mark.gpu


def scaled(u, s):
    """Density, momentum and energy by one factor: the same velocities."""
    return np.ascontiguousarray(u * s)


def low_words_of_ones(u):
    """Densities whose low 32 bits are ones (no rounded reciprocal is taken)."""
    v = np.ascontiguousarray(u.copy())
    v[0].view(np.uint64)[...] |= np.uint64(0xFFFFFFFF)
    return v


def supersonic(u, mach):
    """The whole field moving at `mach` times its largest sound speed along
    both axes: the state outside the wave is sampled."""
    r, p = u[0], 0.4 * (u[3] - 0.5 * (u[1] ** 2 + u[2] ** 2) / u[0])
    c = mach * float(np.sqrt(1.4 * p / r).max())
    m1, m2 = u[1] + r * c, u[2] - r * c
    return np.ascontiguousarray(np.stack([r, m1, m2, p / 0.4 + 0.5 * (m1 ** 2 + m2 ** 2) / r]))


def sonic(u):
    """Exactly sonic uniform columns beside a perturbation: spin and spout at 0."""
    v = np.zeros_like(u)
    c = np.sqrt(1.4)
    v[0], v[1], v[2] = 1.0, c, -c
    v[3] = 1.0 / 0.4 + 0.5 * 2 * 1.4
    v[3, 12:15, 10:14] *= 1.0 + 1e-13
    return v


def momenta(u, exponent):
    """Momenta of 10^exponent and signed zeros: quotients below the range."""
    v = u.copy()
    v[1] = np.where(v[1] > 0, 10.0 ** exponent, -0.0)
    v[2] = np.where(v[2] > 0, -0.0, -(10.0 ** exponent))
    return np.ascontiguousarray(v)


CASES = {
    "smooth": lambda u: u,
    "scale_1e-45": lambda u: scaled(u, 1e-45),
    "scale_1e-36": lambda u: scaled(u, 2.0 ** -122),
    "scale_1e36": lambda u: scaled(u, 2.0 ** 126),
    "scale_1e60": lambda u: scaled(u, 1e60),
    "scale_1e-90": lambda u: scaled(u, 1e-90),
    "low_words_of_ones": low_words_of_ones,
    "supersonic_3": lambda u: supersonic(u, 3.0),
    "supersonic_1": lambda u: supersonic(u, 1.0),
    "sonic": sonic,
    "momenta_1e-80": lambda u: momenta(u, -80),
    "momenta_1e-200": lambda u: momenta(u, -200),
    "momenta_1e-310": lambda u: momenta(u, -310),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("kernels", [("warp", "warp"), ("coop", "march")])
@pytest.mark.parametrize("extra", [{}, {"scheme": 2, "slope_type": 1.5, "gamma": 5.0 / 3.0}])
def test_states_at_the_limits_match_oracle(product_lib, oracle, name, kernels, extra):
    tiny = name.startswith("scale_1e-")
    H = make_params(61, 47, boundary=(1, 2, 3, 1), smallr=1e-120 if tiny else 1e-10, **extra)
    u0 = CASES[name](random_state(61, 47, 41, "smooth"))
    p = orc_from_H(oracle, H)
    want = u0.copy()
    n, dts, t = oracle.run(p, want, 12)
    d = Domain(H, kernels=kernels)
    d.upload(u0)
    d.set_clock()
    d.launch_steps(12)
    got = d.download()
    tg, ng, dt = d.get_clock()
    d.close()
    assert ng == n == 12 and dt == dts[-1] and tg == t
    assert np.isfinite(want).all()
    assert bitwise_equal(got, want), describe_mismatch(got, want)


@pytest.mark.parametrize("gamma", [1.0001, 300.0])
def test_gamma_beyond_the_fast_range(product_lib, oracle, gamma):
    H = make_params(40, 33, gamma=gamma)
    u0 = random_state(40, 33, 43, "smooth", gamma)
    p = orc_from_H(oracle, H)
    want = u0.copy()
    oracle.run(p, want, 6)
    d = Domain(H)
    d.upload(u0)
    d.set_clock()
    d.launch_steps(6)
    got = d.download()
    d.close()
    assert bitwise_equal(got, want), describe_mismatch(got, want)
