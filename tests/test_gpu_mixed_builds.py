"""The FP32-mixed 2D stage kernel exists in two builds, for four and for five CTAs per
SM; the grid's 16x8 tiles choose (more than one round of four: five).  A state
repeated in the periodic y direction must step to the repeated result, bit for bit:
the one copy with the first build, the three copies with the second, whole tiles and
ragged ones, between walls in x and periodic."""
import dataclasses

import numpy as np
import pytest

from helpers import smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wall,limiter", [(False, "mc"), (True, "minmod")])
@pytest.mark.parametrize("nx,ny", [(608, 64), (611, 50), (1000, 37)])
def test_repeated_state(cuda_lib, nx, ny, wall, limiter):
    import torch

    from openmhd_gb300 import Solver, flip, orszag_tang

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = [-(-nx // 16) * -(-n // 8) for n in (ny, 3 * ny)]
    if not tiles[0] <= 4 * sms < tiles[1]:
        pytest.skip("the line lies elsewhere on this device")
    one, _ = orszag_tang(nx, ny, precision="mixed", limiter=limiter)
    if wall:
        one = dataclasses.replace(one, bc_kind=(1, 1, 0, 0, 0, 0), bc_flip=(flip(1, 6), flip(1, 6), 0, 0, 0, 0))
    three = dataclasses.replace(one, jx=3 * ny + 2)
    U = smooth_state(one.jx, one.ix, nx)
    U[:, 0], U[:, -1] = U[:, -2], U[:, 1]
    V = np.concatenate([U[:, :1]] + 3 * [U[:, 1:-1]] + [U[:, -1:]], axis=1)
    res = []
    for cfg, state in ((one, U), (three, V)):
        s = Solver(cfg).put_state(state)
        s.step(3)
        assert s.sync().status == 0
        res.append(s.get_state_numpy())
    for k in range(3):
        part = res[1][:, 1 + k * ny : 1 + (k + 1) * ny]
        assert np.array_equal(part, res[0][:, 1:-1]), k
