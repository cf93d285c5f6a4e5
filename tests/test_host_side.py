"""The library's host code where a call is refused or a context goes away, and
the kernels it launches for a choice, on a stand-in for the CUDA runtime
(_fake_device.py): no device is touched."""
import pytest

from hydro_b200 import Domain, HydroB200Error, _lib, make_params
import _fake_device


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return _fake_device.build(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def lib(fake, monkeypatch):
    monkeypatch.setattr(_lib, "_lib", fake)
    fake.fake_refuse(b"")
    fake.fake_launched(), fake.fake_faults()
    return fake


@pytest.mark.parametrize("precision", ["fp64", "fma", "mixed"])
def test_a_refused_list_launch_leaves_no_list_behind(lib, precision):
    """The cooperative sweep's first launch lists windows, its second works the
    list and empties it.  Where the second is refused the list is emptied all
    the same, so that no later sweep appends to it beyond its room."""
    d = Domain(make_params(300, 200), precision=precision, kernels=("coop", "coop"))
    lib.fake_refuse(b"coop_")
    for k in range(4):
        with pytest.raises(HydroB200Error):
            d.godunov(1 + k % 2, 1e-6)
    lib.fake_refuse(b"")
    d.godunov(1, 1e-6)
    d.close()
    assert lib.fake_faults() == b""


def test_the_maxima_s_host_memory_goes_with_its_context(lib):
    """The words the Courant maxima are written to lie in a page that outlives
    one domain.  After a reset of the device the page is gone: the next
    context's domains have one of their own, and domains of one context share
    theirs."""
    H = make_params(30, 20)
    for _ in range(3):
        doms = [Domain(H) for _ in range(3)]
        assert {d.courant() for d in doms} == {(2.0, 2.0)}
        for d in doms:
            d.close()
        d = Domain(H)
        assert d.courant() == (2.0, 2.0)
        d.close()
        assert lib.fake_pages() == 1
        lib.fake_reset()
    assert lib.fake_faults() == b""
