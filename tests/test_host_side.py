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


def swept(lib, d):
    lib.fake_launched()
    d.godunov(1, 1e-6)
    return [k for k, _ in _fake_device.launched(lib)]


# Mixed x kernels of a grid of few windows: two-cell windows, marching rows.
@pytest.mark.parametrize("x,kx", [("warp", "xcell_mixed_kernel"), ("march", "sweep_mixed_kernel"),
                                  ("bulk", "xpipe_mixed_kernel"), (None, "xcell1_mixed_kernel")])
@pytest.mark.parametrize("y,ky", [("march", "sweep_mixed_kernel"), (None, "ycell_mixed_kernel")])
@pytest.mark.parametrize("nx,ny", [(30, 20), (512, 512)])
def test_small_mixed_grids_run_the_kernel_that_was_chosen(lib, nx, ny, x, kx, y, ky):
    """One cell per lane is the default's choice on small grids, and only that:
    a kernel that the caller names is the one that runs, and "auto" gives the
    default back."""
    d = Domain(make_params(nx, ny), precision="mixed")
    assert swept(lib, d) == ["xcell1_mixed_kernel", "ycell_mixed_kernel"]
    d.set_kernels(x, y)
    assert swept(lib, d) == [kx, ky]
    if x in ("warp", "march"):
        e = Domain(make_params(nx, ny), precision="mixed",
                   xsweep={"warp": "cell", "march": "march"}[x])
        assert swept(lib, e) == [kx, "ycell_mixed_kernel"]
        e.close()
    d.set_kernels("auto", "auto")
    assert swept(lib, d) == ["xcell1_mixed_kernel", "ycell_mixed_kernel"]
    # A captured pair of steps is captured anew for another choice.
    d.launch_steps(2)
    assert "xcell1_mixed_kernel" in [k for k, _ in _fake_device.launched(lib)]
    d.set_kernels("warp", "march")
    d.launch_steps(2)
    names = [k for k, _ in _fake_device.launched(lib)]
    assert "xcell_mixed_kernel" in names and "xcell1_mixed_kernel" not in names
    assert "sweep_mixed_kernel" in names and "ycell_mixed_kernel" not in names
    d.close()


def test_larger_mixed_grids_keep_two_cells_a_lane(lib):
    d = Domain(make_params(513, 512), precision="mixed")
    assert swept(lib, d) == ["xcell_mixed_kernel", "sweep_mixed_kernel"]
    d.close()


@pytest.mark.parametrize("precision", ["fp64", "fma"])
@pytest.mark.parametrize("kernel", ["warp", "coop", "auto"])
@pytest.mark.parametrize("nx,ny", [(3, 3600000), (3600000, 3)])
def test_long_lines_are_launched(lib, precision, kernel, nx, ny):
    """Lines of more windows than a launch grid's y extent holds CTAs."""
    d = Domain(make_params(nx, ny), precision=precision, kernels=(kernel, kernel))
    d.godunov(1, 1e-9)
    d.close()
