"""The Courant maxima after the device clock has stopped before some of the steps
that were launched, by nstepmax or by tend, on an even or an odd step, captured
in step pairs or one by one: they are the state's own, and a run taken up again
from there is the unbroken run."""
import pytest

from hydro_b200 import Domain, make_params
from _helpers import bitwise_equal, random_state

pytestmark = pytest.mark.gpu

NX, NY, STEPS = 50, 40, 12


def domain(precision, one_by_one, u):
    d = Domain(make_params(NX, NY), precision=precision)
    d.profile(one_by_one)  # sweeps that are timed are not replayed in pairs
    d.upload(u)
    d.set_clock()
    return d


@pytest.mark.parametrize("precision", ["fp64", "fma", "mixed"])
@pytest.mark.parametrize("one_by_one", [False, True])
@pytest.mark.parametrize("by", ["nstepmax", "tend"])
@pytest.mark.parametrize("stop", [1, 4, 5])
@pytest.mark.parametrize("launched", [6, 7, 10])
@pytest.mark.parametrize("look", [False, True])
def test_stopped_before_the_last_launched_step(precision, one_by_one, by, stop, launched, look):
    u0 = random_state(NX, NY, 1, "smooth")
    whole = domain(precision, one_by_one, u0)
    whole.reserve_dts(STEPS)
    whole.set_clock()
    whole.launch_steps(STEPS)
    dts = whole.get_dts(STEPS)
    limit = {"nstepmax": stop} if by == "nstepmax" else {"tend": float(dts[:stop].sum()) - 1e-12}

    d = domain(precision, one_by_one, u0)
    d.launch_steps(launched, **limit)
    if look:
        fresh = Domain(make_params(NX, NY), precision=precision)
        fresh.upload(d.download())
        assert d.courant() == fresh.courant()
        fresh.close()
    t, n, dt = d.get_clock()
    assert n == stop
    if look:
        assert d.courant()[0] > 0.1
    d.set_clock(t, n, dt)
    d.launch_steps(STEPS - stop)
    assert d.get_clock() == whole.get_clock()
    assert d.courant() == whole.courant()
    assert bitwise_equal(d.download(), whole.download())
    d.close()
    whole.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_an_odd_step_that_no_even_step_precedes(precision):
    """Its maxima hold nothing of the state before it."""
    H = make_params(NX, NY)
    u = random_state(NX, NY, 2, "smooth")
    u[1:3] *= 20.0
    u[3] += 300.0
    d = Domain(H, precision=precision)
    d.upload(u)
    fast = d.courant()
    d.set_clock(0.0, 3, 1e-9)
    d.upload(random_state(NX, NY, 1, "smooth"))
    d.launch_steps(1)
    fresh = Domain(H, precision=precision)
    fresh.upload(d.download())
    assert d.courant() == fresh.courant()
    assert fresh.courant()[0] < 0.5 * fast[0]
