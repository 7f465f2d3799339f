"""A gradient that is infinite or NaN in one cell reaches the cells whose values that
cell's result depends on, and no others: a slope does not depend on the neighbour that
its limiter did not select."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limiter", ["minmod", "mc"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("side", [-1, 1])
def test_nonfinite_gradient_stays_within_the_stencil(cuda_lib, limiter, bad, side):
    """Every primitive variable grows with slopes that fall off towards one side in x, so
    that every limiter selects the difference on that side and a cell's flux difference
    reads one cell on the other side (two with both differences): after the two stages
    of a step nothing beyond two cells there.  The slopes fall by a factor of two a cell
    (minmod takes the smaller) or of five (MC: its central slope, (gA + gB) / 4, is
    larger than gB where gB < gA / 3), within eight cells of the bad one."""
    import torch

    from openmhd_gb300 import SolverConfig
    from openmhd_gb300.adjoint import AdjointRun

    nx, ny, c = 40, 12, 20  # the cell of the bad gradient, in x
    cfg = SolverConfig(nd=2, ix=nx + 2, jx=ny + 2, dx=1.0, dy=1.0, cfl=0.01, limiter=limiter,
                       bc_kind=(1, 1, 0, 0, 0, 0), bc_flip=(0,) * 6)
    ratio = 2.0 if limiter == "minmod" else 5.0
    ramp = 1 - ratio ** -(8.0 + np.clip(side * (np.arange(nx + 2) - c), -8, 8))
    w = [m + a * ramp for m, a in ((0.3, 0.1), (0.2, 0.07), (0.1, 0.05), (1.0, 0.2), (1.5, 0.3), (0.5, 0.1), (0.4, 0.08),
                                   (0.3, 0.06), (0.1, 0.04))]  # vx vy vz p rho Bx By Bz psi
    vx, vy, vz, p, ro, bx, by, bz, ps = (np.broadcast_to(a, (ny + 2, nx + 2)) for a in w)
    en = 0.5 * (ro * (vx**2 + vy**2 + vz**2) + bx**2 + by**2 + bz**2) + p / (cfg.gamma - 1)
    U = torch.from_numpy(np.stack([ro * vx, ro * vy, ro * vz, en, ro, bx, by, bz, ps])).cuda()
    run = AdjointRun(cfg, 1, 1)
    run.forward(U)
    for var in range(9):
        g = torch.zeros(cfg.shape, dtype=torch.float64, device="cuda")
        g[var, ny // 2, c] = bad
        out = run.backward(g).cpu().numpy()
        run.sync()
        hit = side * (np.nonzero(~np.isfinite(out).all(axis=(0, 1)))[0] - c)  # columns, counted along the side
        assert 0 in hit
        assert hit.min() >= -2 and hit.max() <= 4, (var, hit)
