"""Which states the 3D stage kernels refuse does not depend on where they cut the grid
into z chunks (pick_zchunk): a column of tiles alone (short chunks), and the same state
repeated 40 times in y (long ones), end with the same status."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NZ = 130


def _status(cfg, U):
    from openmhd_gb300 import Solver
    from openmhd_gb300.solver import OmhdError

    s = Solver(cfg)
    try:
        s.put_state(U)
        s.step(1)
        s.sync()
    except OmhdError as e:
        return e.code
    return 0


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_parity"])
@pytest.mark.parametrize("kind", ["nan", "tiny pressure", "negative pressure"])
def test_status_does_not_depend_on_the_cut(cuda_lib, precision, kind):
    from openmhd_gb300 import field_loop3d

    one, _ = field_loop3d(32, 8, NZ, precision=precision, limiter="mc")
    many = dataclasses.replace(one, jx=8 * 40 + 2)
    rng = np.random.default_rng(1)
    n = one.shape[1:]
    ro, p = 1 + 0.1 * rng.random(n), 0.6 + 0.05 * rng.random(n)
    zero = np.zeros(n)
    base = np.stack([zero, zero, zero, p / (one.gamma - 1), ro, zero, zero, zero, zero])
    for k in (1, 2, 7, 20, 63, 64, 65, 66, 100, 129):
        U = base.copy()
        U[3, k, 4, 16] = {"nan": np.nan, "tiny pressure": 1e-50, "negative pressure": -1.0}[kind]
        V = np.concatenate([U[:, :, :1]] + 40 * [U[:, :, 1:-1]] + [U[:, :, -1:]], axis=2)
        a, b = _status(one, U), _status(many, V)
        assert a == b, (k, a, b)
        assert a == 1 or kind != "negative pressure"
