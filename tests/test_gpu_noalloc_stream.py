"""Allocation-free steps that follow one another on a stream, without a wait
between them, and with the caller's own work between them: each takes the state
that the one before left."""
import ctypes as C

import pytest
import torch

from hydro_b200 import HydroRun, load, make_params
from hydro_b200._lib import HB_OK
from _helpers import bitwise_equal, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("between", ["nothing", "kernel", "copy", "event", "memset"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (64, 64), (250, 125), (64, 4000)])
def test_steps_in_a_row(product_lib, nx, ny, between):
    H = make_params(nx, ny)
    u0 = random_state(nx, ny, nx, "smooth")
    dt, steps = 0.1 / nx, 8
    ref = HydroRun(H, u0.copy())
    lib = load()
    state = torch.from_numpy(u0).to("cuda:0")
    spare = torch.empty_like(state)
    main, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(main):
        for k in range(steps):
            assert lib.hydro_b200_godunov_noalloc(C.byref(H), state.data_ptr(), 1 + k % 2, dt,
                                                  C.c_void_p(main.cuda_stream)) == HB_OK
            if between == "kernel":  # reads and writes what the step left
                state[0] *= 1.25
            elif between == "copy":
                spare.copy_(state)
                state.copy_(spare)
            elif between == "memset":
                state[2].zero_()
            elif between == "event":
                other.wait_stream(main)
                with torch.cuda.stream(other):
                    state[0] *= 1.25
                main.wait_stream(other)
    torch.cuda.synchronize()
    for k in range(steps):
        ref.godunov(1 + k % 2, dt)
        u = ref.sync_to_host()
        if between in ("kernel", "event"):
            u[0] *= 1.25
        elif between == "memset":
            u[2] = 0.0
        ref.sync_to_device()
    want = ref.uold.copy()
    ref.close()
    assert bitwise_equal(state.cpu().numpy(), want)
