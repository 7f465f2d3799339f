"""The pipelined FP64 2D kernel cuts the grid into tiles of 4 to 16 rows depending
on its size (pick_rows): every height, ragged or not, walls or periodic, minmod or
MC, must give the oracle's step."""
import dataclasses

import pytest

from helpers import assert_parity, smooth_state

pytestmark = pytest.mark.gpu


def _rows(nx, ny, nsm=152):
    """The kernel's rule, restated: the rows of a tile for an nx x ny grid."""
    ntx = -(-nx // 16)
    return min(range(16, 3, -1), key=lambda ty: -(-ntx * -(-ny // ty) // nsm) * (ty + 4.7))


# one grid per tile height the rule can give (checked below), ragged in x and y
GRIDS = [(36, 32), (66, 125), (250, 54), (330, 47), (650, 23), (500, 36), (416, 47), (90, 257), (500, 46), (196, 137),
         (410, 66), (500, 57), (330, 106), (2, 2), (17, 5)]


def test_grids_cover_the_heights():
    assert {_rows(nx, ny) for nx, ny in GRIDS} == set(range(4, 17))


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("wall,limiter", [(False, "mc"), (True, "minmod")])
def test_step_vs_oracle(cuda_lib, oracle_mod, nx, ny, wall, limiter):
    from openmhd_gb300 import Solver, flip, orszag_tang
    from oracle.oracle import Grid

    cfg, _ = orszag_tang(nx, ny, precision="fp64", limiter=limiter)
    if wall:
        cfg = dataclasses.replace(cfg, bc_kind=(1, 1, 1, 1, 0, 0),
                                  bc_flip=(flip(1, 6), flip(1, 6), flip(2, 7), flip(2, 7), 0, 0))
    s = Solver(cfg).put_state(smooth_state(cfg.jx, cfg.ix, nx))
    g = Grid.from_solver_config(cfg, omp=True)
    g.U[...] = s.get_state_numpy()
    s.step(1)
    assert s.sync().status == 0
    g.step(1)
    assert_parity(s.get_state_numpy(), g.U, 1e-12, f"{nx}x{ny}")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(36, 12), (333, 50), (500, 57), (170, 19)])
def test_resistive_step_vs_oracle(cuda_lib, oracle_mod, nx, ny, precision):
    """Resistive reconnection between symmetry walls: the field copies of the
    pipelined kernel and the tabulated resistivity."""
    from openmhd_gb300 import Solver, reconnection2d
    from openmhd_gb300.metrics import scaled_l1
    from oracle.oracle import Grid

    cfg, model = reconnection2d(nx, ny, precision=precision)
    s = Solver(cfg).init_model(model)
    g = Grid.from_solver_config(cfg, omp=True)
    g.U[...] = s.get_state_numpy()
    s.step(2)
    assert s.sync().status == 0
    g.step(2)
    if precision == "fp64":
        assert_parity(s.get_state_numpy(), g.U, 1e-11, f"{nx}x{ny}")
    else:  # the mixed path's own bound over a few steps
        assert scaled_l1(s.get_state_numpy(), g.U).max() <= 1e-6
