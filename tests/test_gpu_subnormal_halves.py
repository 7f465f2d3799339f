"""The halving of the second stage (rk_tvd22) keeps numbers below 2^-1022: a uniform
state, whose flux differences vanish, stays as it is to the last bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_parity"])
@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("value", [5e-324, 1e-320, -1e-310, 2.0**-1023, 2.0**-1022, -(2.0**-1021), 3e-308, 0.0, 1e-300])
def test_uniform_state_is_kept(cuda_lib, precision, nd, value):
    from openmhd_gb300 import Solver, field_loop3d, orszag_tang

    cfg = (orszag_tang(40, 24, precision=precision) if nd == 2 else field_loop3d(20, 12, 9, precision=precision))[0]
    U = np.zeros(cfg.shape)
    U[2], U[3], U[4], U[5], U[6], U[7] = value, 2.0, 1.0, 0.25, value, value  # mz, E, rho, Bx, By, Bz
    s = Solver(cfg).put_state(U)
    s.step(3)
    assert s.sync().status == 0
    got = s.get_state_numpy()
    assert np.array_equal(got.view(np.int64), U.view(np.int64))
