"""The 3D stage kernels cut the grid into z chunks whose length depends on the
grid's size (pick_zchunk): results must not depend on the cut, and grids of any
depth must give the oracle's step."""
import dataclasses

import numpy as np
import pytest

from helpers import assert_parity

pytestmark = pytest.mark.gpu


def _state(cfg, seed):
    """Mild random state: every HLLD branch near the sound speed, no negative pressure."""
    rng = np.random.default_rng(seed)
    n = cfg.shape[1:]
    f = lambda mean, amp: mean + amp * rng.uniform(-1, 1, n)  # noqa: E731
    ro, p, v, B = f(1.0, 0.1), f(0.6, 0.05), [f(0.3, 0.2) for _ in range(3)], [f(0.2, 0.2) for _ in range(3)]
    en = 0.5 * (ro * sum(a * a for a in v) + sum(b * b for b in B)) + p / (cfg.gamma - 1)
    return np.stack([ro * v[0], ro * v[1], ro * v[2], en, ro, *B, f(0.0, 0.01)])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nz", [5, 64, 65, 130])
def test_result_does_not_depend_on_the_cut(cuda_lib, precision, nz):
    """A grid of one column of CTAs, and the same state repeated 40 times along
    the periodic y axis (40 columns: other chunks): the same bits in every copy."""
    from openmhd_gb300 import Solver, field_loop3d

    cfg, _ = field_loop3d(32, 8, nz, precision=precision)
    big = dataclasses.replace(cfg, jx=8 * 40 + 2)
    U = _state(cfg, 3)
    Ub = np.concatenate([U[:, :, :1], np.tile(U[:, :, 1:-1], (1, 1, 40, 1)), U[:, :, -1:]], axis=2)
    a, b = Solver(cfg).put_state(U), Solver(big).put_state(Ub)
    a.step(2)
    b.step(2)
    assert a.sync().status == 0 and b.sync().status == 0
    ra, rb = a.get_state_numpy()[:, 1:-1, 1:-1, 1:-1], b.get_state_numpy()[:, 1:-1, 1:-1, 1:-1]
    assert np.array_equal(rb, np.tile(ra, (1, 1, 40, 1)))


@pytest.mark.parametrize("wall", [False, True])
@pytest.mark.parametrize("nz", [2, 3, 64, 67])
def test_any_depth_vs_oracle(cuda_lib, oracle_mod, nz, wall):
    from openmhd_gb300 import Solver, field_loop3d, flip
    from oracle.oracle import Grid

    cfg, _ = field_loop3d(33, 9, nz, precision="fp64", limiter="mc")
    if wall:
        f = flip(3, 8)  # mz, Bz
        cfg = dataclasses.replace(cfg, bc_kind=(0, 0, 0, 0, 1, 1), bc_flip=(0, 0, 0, 0, f, f), eta="harris_xz")
    s = Solver(cfg).put_state(_state(cfg, nz))
    g = Grid.from_solver_config(cfg, omp=True)
    g.U[...] = s.get_state_numpy()
    s.step(1)
    assert s.sync().status == 0
    g.step(1)
    assert_parity(s.get_state_numpy(), g.U, 1e-12, f"nz {nz}")
