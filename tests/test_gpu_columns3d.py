"""The FP64 3D stage kernel marches 16x16 columns or pairs of 16x8 columns, whichever the
grid's size makes cheaper, each with a warp that owns no cells: grids of either kind,
ragged in x and y, periodic or with walls and resistivity, against the oracle's step."""
import dataclasses

import numpy as np
import pytest

from helpers import assert_parity

pytestmark = pytest.mark.gpu

GRIDS = [(49, 65, 8), (97, 33, 8), (48, 64, 8), (35, 23, 5)]


def _pairs(nx, ny, nz, resistive, nsm=152):
    """The rule, restated: whether the grid is cut into pairs of 16x8 columns."""
    cost = lambda cols, slots: min(-(-cols * -(-nz // c) // slots) * (c + 1.5) for c in range(1, min(nz, 64) + 1))  # noqa: E731
    wide, small = cost(-(-nx // 16) * -(-ny // 16), nsm), cost(-(-nx // 16) * -(-ny // 8), 2 * nsm)
    return (1.11 if resistive else 1.02) * small < wide


def test_grids_cover_both_columns():
    assert {_pairs(*g, r) for g in GRIDS for r in (False, True)} == {False, True}


def _state(cfg, seed):
    """Mild random state: every HLLD branch near the sound speed, no negative pressure."""
    rng = np.random.default_rng(seed)
    n = cfg.shape[1:]
    f = lambda mean, amp: mean + amp * rng.uniform(-1, 1, n)  # noqa: E731
    ro, p, v, B = f(1.0, 0.1), f(0.6, 0.05), [f(0.3, 0.2) for _ in range(3)], [f(0.2, 0.2) for _ in range(3)]
    en = 0.5 * (ro * sum(a * a for a in v) + sum(b * b for b in B)) + p / (cfg.gamma - 1)
    return np.stack([ro * v[0], ro * v[1], ro * v[2], en, ro, *B, f(0.0, 0.01)])


@pytest.mark.parametrize("nx,ny,nz", GRIDS)
@pytest.mark.parametrize("wall", [False, True])
def test_step_vs_oracle(cuda_lib, oracle_mod, nx, ny, nz, wall):
    from openmhd_gb300 import Solver, field_loop3d, flip
    from oracle.oracle import Grid

    cfg, _ = field_loop3d(nx, ny, nz, precision="fp64", limiter="minmod" if wall else "mc")
    if wall:
        f = [flip(1, 6), flip(2, 7), flip(3, 8)]
        cfg = dataclasses.replace(cfg, bc_kind=(1,) * 6, bc_flip=(f[0], f[0], f[1], f[1], f[2], f[2]), eta="harris_xz")
    s = Solver(cfg).put_state(_state(cfg, nx))
    g = Grid.from_solver_config(cfg, omp=True)
    g.U[...] = s.get_state_numpy()
    s.step(1)
    assert s.sync().status == 0
    g.step(1)
    assert_parity(s.get_state_numpy(), g.U, 1e-12, f"{nx}x{ny}x{nz}")


@pytest.mark.parametrize("nx,ny,nz", [(40, 8, 6), (33, 7, 70), (48, 6, 5)])
@pytest.mark.parametrize("wall", [False, True])
def test_mixed_columns_agree(cuda_lib, nx, ny, nz, wall):
    """FP32-mixed: a grid of 32x8 columns, and its state repeated five times along the
    periodic y axis, which 16x16 columns cover in fewer: the same bits in every copy."""
    from openmhd_gb300 import Solver, field_loop3d, flip

    columns = lambda n: (-(-nx // 32) * -(-n // 8), -(-nx // 16) * -(-n // 16))  # noqa: E731
    assert columns(ny)[0] <= columns(ny)[1] and columns(5 * ny)[0] > columns(5 * ny)[1]
    one, _ = field_loop3d(nx, ny, nz, precision="mixed", limiter="mc")
    if wall:
        f = [flip(1, 6), flip(3, 8)]
        one = dataclasses.replace(one, bc_kind=(1, 1, 0, 0, 1, 1), bc_flip=(f[0], f[0], 0, 0, f[1], f[1]))
    five = dataclasses.replace(one, jx=5 * ny + 2)
    U = _state(one, ny)
    U[:, :, 0], U[:, :, -1] = U[:, :, -2], U[:, :, 1]
    V = np.concatenate([U[:, :, :1]] + 5 * [U[:, :, 1:-1]] + [U[:, :, -1:]], axis=2)
    res = []
    for cfg, state in ((one, U), (five, V)):
        s = Solver(cfg).put_state(state)
        s.step(2)
        assert s.sync().status == 0
        res.append(s.get_state_numpy())
    for k in range(5):
        assert np.array_equal(res[1][:, :, 1 + k * ny : 1 + (k + 1) * ny], res[0][:, :, 1:-1]), k
