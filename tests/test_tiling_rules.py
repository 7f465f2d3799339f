"""How the stage kernels cut a grid, as the library itself answers (omhd_probe_tiling),
against the rules restated here; needs no GPU."""
import ctypes as C
import itertools

import pytest

from test_gpu_columns3d import GRIDS as COLUMN_GRIDS
from test_gpu_tile_rows import GRIDS as ROW_GRIDS

SMS = [1, 78, 132, 148, 152, 160]


@pytest.fixture(scope="module")
def tiling():
    from openmhd_gb300 import _lib
    from openmhd_gb300.build import build

    build()
    lib = _lib.load()

    def of(cfg, sms):
        c, t = cfg.to_c(), (C.c_int * 4)()
        assert lib.omhd_probe_tiling(C.byref(c), sms, t) == 0
        return tuple(t)

    of.lib = lib
    return of


def _cfg(n, precision, resistive=False, **k):
    from openmhd_gb300 import SolverConfig

    ix, jx, kx = [v + 2 for v in n] + [1] * (3 - len(n))
    eta = ("recon2d" if len(n) == 2 else "harris_xz") if resistive else "none"
    return SolverConfig(nd=len(n), ix=ix, jx=jx, kx=kx, precision=precision, eta=eta, **k)


def _up(a, b):
    return -(-a // b)


def _zchunk(columns, nz, slots):
    """(cost, planes): the fewest rounds x (planes + 1.5), the longest chunk among equals."""
    best = min((_up(columns * _up(nz, c), slots) * (c + 1.5), -c) for c in range(1, min(nz, 64) + 1))
    return best[0], -best[1]


def _columns(n, tx, ty, ctas, sms):
    cost, tz = _zchunk(_up(n[0], tx) * _up(n[1], ty), n[2], ctas * sms)
    return cost, (tx, ty, tz, ctas)


@pytest.mark.parametrize("sms", SMS)
@pytest.mark.parametrize("resistive", [False, True])
def test_rows_of_a_pipelined_tile(tiling, sms, resistive):
    for n in ROW_GRIDS + [(64, 64), (256, 256), (500, 125), (999, 501), (4096, 2048), (1000, 8), (8, 1000)]:
        ntx = _up(n[0], 16)
        rows = min(range(16, 3, -1), key=lambda ty: _up(ntx * _up(n[1], ty), sms) * (ty + 4.7))
        for lm in ("minmod", "mc"):
            assert tiling(_cfg(n, "fp64", resistive, limiter=lm), sms) == (16, rows, 1, 1), n
        assert tiling(_cfg(n, "fp64", resistive, limiter="koren"), sms) == (16, 16, 1, 1)
        assert tiling(_cfg(n, "fp64", resistive, flux="hll"), sms) == (16, 16, 1, 1)


def test_row_grids_take_every_height(tiling):
    assert {tiling(_cfg(n, "fp64"), 152)[1] for n in ROW_GRIDS} == set(range(4, 17))


@pytest.mark.parametrize("sms", SMS)
def test_mixed_2d_builds(tiling, sms):
    for n in [(64, 64), (256, 256), (608, 64), (608, 192), (611, 50), (1000, 37), (1000, 111), (4096, 2048), (2432, 32)]:
        tiles = _up(n[0], 16) * _up(n[1], 8)
        assert tiling(_cfg(n, "mixed"), sms) == (16, 8, 1, 5 if tiles > 4 * sms else 4)
        assert tiling(_cfg(n, "mixed", flux="hll"), sms) == (16, 8, 1, 4)


GRIDS_3D = COLUMN_GRIDS + [(64, 32, 64), (256, 128, 256), (100, 100, 200), (512, 256, 512), (64, 64, 128), (33, 9, 2), (2, 2, 2),
                           (16, 16, 700), (128, 128, 8), (8, 128, 128)]


@pytest.mark.parametrize("sms", SMS)
@pytest.mark.parametrize("resistive", [False, True])
def test_columns_3d_fp64(tiling, sms, resistive):
    for n in GRIDS_3D:
        (wide, a), (small, b) = _columns(n, 16, 16, 1, sms), _columns(n, 16, 8, 2, sms)
        want = b if (1.11 if resistive else 1.02) * small < wide else a
        assert tiling(_cfg(n, "fp64", resistive), sms) == want, n
        default = _columns(n, 32, 8, 1, sms)[1]
        assert tiling(_cfg(n, "fp64", resistive, flux="hllc"), sms) == default
        assert tiling(_cfg(n, "fp64_parity", resistive), sms) == default


@pytest.mark.parametrize("sms", SMS)
@pytest.mark.parametrize("resistive", [False, True])
def test_columns_3d_mixed(tiling, sms, resistive):
    """Also thin grids, of which 16x16 columns would leave half outside: never the column
    with the higher cost."""
    thin = [(1024, 8, 1024), (512, 8, 512), (512, 24, 512), (512, 40, 512), (128, 8, 128), (300, 72, 300), (700, 8, 50)]
    for n in GRIDS_3D + thin:
        (square, a), (flat, b) = _columns(n, 16, 16, 2, sms), _columns(n, 32, 8, 2, sms)
        if resistive:
            want = a if square <= flat else b
        else:
            want = a if _up(n[0], 16) * _up(n[1], 16) < _up(n[0], 32) * _up(n[1], 8) else b
        got = tiling(_cfg(n, "mixed", resistive), sms)
        assert got == want, n
        assert (square if got[0] == 16 else flat) == min(square, flat), n
        assert tiling(_cfg(n, "mixed", resistive, flux="llf"), sms) == b
    if sms == 152 and resistive:
        assert all(tiling(_cfg(n, "mixed", True), sms)[:2] == (32, 8) for n in thin)


def test_column_grids_take_both(tiling):
    assert {tiling(_cfg(n, "fp64", r), 152)[1] for n, r in itertools.product(COLUMN_GRIDS, (False, True))} == {8, 16}


def test_bad_arguments(tiling):
    c, t = _cfg((64, 64), "fp64").to_c(), (C.c_int * 4)()
    assert tiling.lib.omhd_probe_tiling(C.byref(c), 0, t) == 4
    assert tiling.lib.omhd_probe_tiling(C.byref(c), 152, None) == 4
    assert tiling.lib.omhd_probe_tiling(None, 152, t) == 4
    c.ix = 3
    assert tiling.lib.omhd_probe_tiling(C.byref(c), 152, t) == 4


@pytest.mark.gpu
def test_gpu_grids_cover_the_rules_on_this_device(tiling, cuda_lib):
    """The grids that the GPU tests step through reach every tile height and both columns
    with this device's SM count."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert {tiling(_cfg(n, "fp64"), sms)[1] for n in ROW_GRIDS} >= {4, 16}
    assert len({tiling(_cfg(n, "fp64"), sms)[1] for n in ROW_GRIDS}) >= 8
    assert {tiling(_cfg(n, "fp64", r), sms)[1] for n, r in itertools.product(COLUMN_GRIDS, (False, True))} == {8, 16}
