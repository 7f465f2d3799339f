"""The CFL maximum found through binary32 upper bounds (cfl_upper): dt after a step
is the FP64 maximum over all cells of the new state, bit for bit what a kernel that
evaluates every cell finds -- for states whose maximum hides in one cell, ties
everywhere, low beta, high Mach number and scales outside binary32."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(cfg, kind, seed):
    rng = np.random.default_rng(seed)
    n = cfg.shape[1:]
    one = np.ones(n)
    noise = lambda a: 1 + a * rng.uniform(-1, 1, n)  # noqa: E731
    ro, p, v, B = one.copy(), 0.5 * one, [0.2 * one] * 3, [0.3 * one] * 3
    scale = 1.0
    if kind == "ties":
        pass
    elif kind == "one_cell":
        p = p * noise(1e-3)
        p[tuple(k // 2 for k in n)] *= 1.004
    elif kind == "near_ties":  # within the bound's margin of one another
        p = p * noise(1e-6)
    elif kind == "low_beta":
        p, B = 1e-4 * noise(0.5), [b * noise(1e-5) for b in B]
    elif kind == "high_mach":
        p, v = 1e-4 * noise(0.5), [2.0 * noise(1e-4) for _ in v]
    elif kind == "degenerate":  # gamma p = B^2 = Bn^2: the discriminant vanishes
        B = [np.sqrt(5.0 / 3.0 * 0.5) * noise(1e-9), 1e-9 * noise(1.0), 0 * one]
    else:  # powers of ten outside binary32
        scale = 10.0 ** float(kind)
        p = p * noise(0.3)
    r = ro * scale
    B = [b * np.sqrt(scale) for b in B]
    p = p * scale
    en = 0.5 * (r * sum(a * a for a in v) + sum(b * b for b in B)) + p / (cfg.gamma - 1)
    return np.stack([r * v[0], r * v[1], r * v[2], en, r, *B, 0 * one])


def _speed(U, gamma, nd):
    """Largest |v| + fast speed of the interior, FP64."""
    V = U[(slice(None),) + (slice(1, -1),) * nd]
    v = V[0:3] / V[4]
    B2 = (V[5:8] ** 2).sum(0)
    f1 = gamma * (gamma - 1) * (V[3] - 0.5 * ((v * V[0:3]).sum(0) + B2))
    best = 0.0
    for a in range(nd):
        D = np.maximum((f1 + B2) ** 2 - 4 * f1 * V[5 + a] ** 2, 0)
        best = max(best, (np.abs(v[a]) + np.sqrt((f1 + B2 + np.sqrt(D)) / (2 * V[4]))).max())
    return best


KINDS = ["ties", "one_cell", "near_ties", "low_beta", "high_mach", "degenerate", "-60", "60"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nd,precision", [(2, "fp64"), (2, "mixed"), (3, "fp64")])
def test_dt_is_the_maximum_over_all_cells(cuda_lib, kind, nd, precision):
    """Grids of many more tiles than the GPU runs at a time, so that most cells are
    decided by their bound (mixed: scales inside binary32 only)."""
    from openmhd_gb300 import Solver, field_loop3d, orszag_tang

    if precision == "mixed" and kind in ("-60", "60"):
        pytest.skip("outside the FP32 face arithmetic")
    if nd == 2:
        cfg, _ = orszag_tang(1000, 1100, precision=precision)
    else:
        cfg, _ = field_loop3d(200, 120, 90, precision=precision)
    cfg = dataclasses.replace(cfg, dx=1.0, dy=1.0, dz=1.0)
    U = _state(cfg, kind, 5)
    s = Solver(cfg).put_state(U)
    first = s.sync().vmax_next
    # 1e-11: rounding of the two formulas' cancellations (low beta: p / E ~ 1e-4)
    want = _speed(s.get_state_numpy(), cfg.gamma, nd)
    assert abs(first - want) <= 1e-11 * want
    for _ in range(2):
        s.step(1)
        info = s.sync()
        want = _speed(s.get_state_numpy(), cfg.gamma, nd)
        assert abs(info.vmax_next - want) <= 1e-11 * want
