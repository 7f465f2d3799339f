"""The CFL maximum is exact whatever cells their bounds leave out (cfl_upper): a small
periodic state, and the same state repeated over a grid of many more tiles than the GPU
runs at a time, most of which are decided by their bound, give the same double and with it
the same dt, at the start and after every step."""
import dataclasses

import numpy as np
import pytest

from test_gpu_cfl_bound import KINDS, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nd,precision", [(2, "fp64"), (2, "mixed"), (3, "fp64"), (3, "mixed")])
def test_maximum_of_a_repeated_state(cuda_lib, kind, nd, precision):
    from openmhd_gb300 import Solver, field_loop3d, orszag_tang

    if precision == "mixed" and kind in ("-60", "60"):
        pytest.skip("outside the FP32 face arithmetic")
    if nd == 2:
        one, times = orszag_tang(48, 32, precision=precision)[0], (30, 20)
    else:
        one, times = field_loop3d(32, 16, 20, precision=precision)[0], (1, 12, 5)
    one = dataclasses.replace(one, dx=1.0, dy=1.0, dz=1.0)
    inner = (slice(None),) + (slice(1, -1),) * nd
    U = _state(one, kind, 11)[inner]
    ghosts = ((0, 0),) + ((1, 1),) * nd
    n = [(s - 2) * t + 2 for s, t in zip(one.shape[1:], times)]
    many = dataclasses.replace(one, ix=n[-1], jx=n[-2], kx=n[0] if nd == 3 else 1)
    a = Solver(one).put_state(np.pad(U, ghosts, mode="wrap"))
    b = Solver(many).put_state(np.pad(np.tile(U, (1,) + times), ghosts, mode="wrap"))
    for step in range(4):
        ia, ib = a.sync(), b.sync()
        assert ia.vmax_next == ib.vmax_next and ia.vmax_next > 0, step
        a.step(1)
        b.step(1)
    assert a.sync().t == b.sync().t
    assert np.array_equal(b.get_state_numpy()[inner], np.tile(a.get_state_numpy()[inner], (1,) + times))
