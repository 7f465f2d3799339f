"""The FP64 products, quotients, roots and differences that the kernels make on the integer pipes
(mul_int, half_exact, div_rn, sqrt_rn, sub_f32 in openmhd_gb300/csrc/omhd_fastmath.h):
against IEEE results on the host, and whole steps in units that reach the ends of their
range, where a face is solved with FP64-pipe products instead."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from helpers import assert_parity

pytestmark = pytest.mark.gpu

TINY = 2.0**-1022


def _probe(lib, a, b):
    import torch

    at, bt = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (a, b))
    out = torch.empty(6 * len(a), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.omhd_probe_mul(C.c_void_p(at.data_ptr()), C.c_void_p(bt.data_ptr()), len(a), C.c_void_p(out.data_ptr())) == 0
    return out.cpu().numpy().reshape(6, -1)


def _significands(rng, n):
    """Random ones and those next to a carry: short, all ones, one bit."""
    m = rng.integers(0, 2**52, n)
    k = n // 4
    m[:k] = rng.integers(0, 16, k)
    m[k : 2 * k] = 2**52 - 1 - rng.integers(0, 16, k)
    m[2 * k : 2 * k + k // 2] = 2 ** rng.integers(0, 52, k // 2)
    return rng.permutation(m)


@pytest.mark.parametrize("lo,hi", [(-60, 60), (-511, 510), (-1022, -400)])
def test_products_equal_ieee(cuda_lib, lo, hi):
    rng = np.random.default_rng(hi + 2000)
    n = 1 << 20
    ab = [np.ldexp(1 + _significands(rng, n) * 2.0**-52, rng.integers(lo, hi + 1, n)) * rng.choice([-1.0, 1.0], n)
          for _ in range(2)]
    for v in ab:
        v[rng.integers(0, n, n // 50)] = rng.choice([0.0, -0.0], n // 50)
    a, b = ab
    got, bad, half = _probe(cuda_lib, a, b)[:3]
    with np.errstate(under="ignore"):
        want, whalf = a * b, a * 0.5
    assert not bad.any()
    tie = _is_tie(a, b)
    normal = np.abs(want) >= 2.0**-1020
    ok = normal & ~tie
    assert np.array_equal(got[ok].view(np.int64), want[ok].view(np.int64))
    # exact ties may round up where IEEE rounds to even: one unit in the last place
    t = normal & tie
    assert np.all(np.abs(np.abs(got[t]).view(np.int64) - np.abs(want[t]).view(np.int64)) <= 1)
    small = ~normal  # subnormal products become signed zeros
    assert np.all(np.abs(got[small] - want[small]) <= 2 * 2.0**-1020)
    assert np.array_equal(np.signbit(got), np.signbit(want))
    keep = (np.abs(a) >= 2 * TINY) | (a == 0)  # exact halves of 2^-1022 or more (the IEEE half may round up to it)
    assert np.array_equal(half[keep].view(np.int64), whalf[keep].view(np.int64))
    assert np.all(half[~keep] == 0) and np.array_equal(np.signbit(half), np.signbit(a))


def _is_tie(a, b):
    """Whether the exact product lies half way between two doubles."""
    ma, mb = (np.frexp(np.abs(v))[0] * 2.0**53 for v in (a, b))
    ia, ib = ma.astype(np.int64), mb.astype(np.int64)
    out = np.zeros(len(a), bool)
    tz = lambda v: np.where(v == 0, 0, np.log2(np.maximum(v & -v, 1))).astype(int)  # noqa: E731
    low = tz(ia) + tz(ib)  # trailing zeros of the 106-bit product
    for i in np.nonzero((low >= 51) & (ia > 0) & (ib > 0))[0]:
        p = int(ia[i]) * int(ib[i])
        s = p.bit_length() - 53
        out[i] = s > 0 and (p & ((1 << s) - 1)) == 1 << (s - 1)
    return out


def test_operands_out_of_range_are_refused(cuda_lib):
    big = [2.0**511, 1.7e308, np.inf, -np.inf, np.nan]
    a = np.array([x for x in big for _ in range(4)] + [2.0**511 - 2.0**458])
    b = np.array([1.0, 0.0, 1e-300, 5e-324] * len(big) + [1.0])
    for u, v in ((a, b), (b, a)):
        bad = _probe(cuda_lib, u, v)[1]
        assert bad[:-1].all() and not bad[-1]
    half = _probe(cuda_lib, np.array([np.inf, -np.inf, np.nan]), np.ones(3))[2]
    assert half[0] == np.inf and half[1] == -np.inf and np.isnan(half[2])


@pytest.mark.parametrize("lo,hi,gap", [(-3, 3, 3), (-125, 128, 40), (-125, -88, 60), (100, 128, 120)])
def test_differences_of_binary32_equal_ieee(cuda_lib, lo, hi, gap):
    """sub_f32: the binary64 difference of two binary32 numbers, bit for bit, over
    operand pairs that cancel, that fill 53 bits and that exceed them, next to
    powers of two, and zeros, infinities and NaN."""
    rng = np.random.default_rng(17)
    n = 1 << 20
    e = rng.integers(lo, hi, n)
    f = np.clip(e + rng.integers(-gap, gap + 1, n), -126, 127)
    m = [(1.0 + (_significands(rng, n) >> 29) / 2.0**23) * rng.choice([-1.0, 1.0], n) for _ in range(2)]
    m[0][: n // 4] = 1.0
    a, b = np.ldexp(m[0], e).astype(np.float32), np.ldexp(m[1], f).astype(np.float32)
    a[-1000:-500] = b[-1000:-500]
    sp = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, 2.0**-126, 3.4e38, -3.4e38], np.float32)
    sa, sb = (v.ravel() for v in np.meshgrid(sp, sp))
    swap = rng.random(n) < 0.5
    a, b = np.where(swap, b, a), np.where(swap, a, b)
    a, b = np.concatenate([a, sa]), np.concatenate([b, sb])
    with np.errstate(invalid="ignore"):
        want = a.astype(np.float64) - b.astype(np.float64)
    got = _probe(cuda_lib, a.astype(np.float64), b.astype(np.float64))[5]
    nan = np.isnan(want)
    assert np.isnan(got[nan]).all()
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


@pytest.mark.parametrize("lo,hi", [(-60, 60), (-1, 1), (-1022, 1023)])
def test_quotients_and_roots_equal_ieee(cuda_lib, lo, hi):
    """Correctly rounded, bit for bit, on exact quotients and squares, their
    neighbours, zeros, subnormals, infinities and NaN."""
    rng = np.random.default_rng(hi)
    n = 1 << 21
    a, b = (np.ldexp(1 + _significands(rng, n) * 2.0**-52, rng.integers(lo, hi + 1, n)) * rng.choice([-1.0, 1.0], n)
            for _ in range(2))
    k = n // 8
    with np.errstate(all="ignore"):
        a[:k] = a[:k] * b[:k]  # near an exact quotient
        a[k : 2 * k] = b[k : 2 * k] ** 2  # near an exact root
        a[2 * k : 3 * k] = np.nextafter(b[2 * k : 3 * k] ** 2, rng.choice([0, np.inf], k))
        special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, TINY, 1.7e308, 1.0])
        for v in (a, b):
            v[rng.integers(0, n, n // 100)] = rng.choice(special, n // 100)
        div, root = _probe(cuda_lib, a, b)[3:5]
        for got, want in ((div, a / b), (root, np.sqrt(a))):
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64))


@pytest.mark.parametrize("ro,pr", [(1.0, 1.0), (1e155, 1e150), (1e-150, 1e-150), (1e-3, 1e149)])
@pytest.mark.parametrize("nd", [2, 3])
def test_steps_in_extreme_units_vs_oracle(cuda_lib, oracle_mod, ro, pr, nd):
    """The step is covariant under a change of units; densities of 1e155 send
    every face to the FP64-pipe products, 1e-150 squares come close to underflow."""
    from openmhd_gb300 import Solver, field_loop3d, orszag_tang
    from oracle.oracle import Grid

    if nd == 2:
        cfg, _ = orszag_tang(40, 24, precision="fp64")
    else:
        cfg, _ = field_loop3d(33, 10, 9, precision="fp64", limiter="mc")
    v0 = np.sqrt(pr / ro)
    rng = np.random.default_rng(7)
    f = lambda mean, amp: mean + amp * rng.uniform(-1, 1, cfg.shape[1:])  # noqa: E731
    r, p = f(1.0, 0.2) * ro, f(0.6, 0.1) * pr
    v, B = [f(0.1, 0.3) * v0 for _ in range(3)], [f(0.1, 0.4) * np.sqrt(pr) for _ in range(3)]
    cfg = dataclasses.replace(cfg, dx=v0 * 0.1, dy=v0 * 0.1, dz=v0 * 0.1)
    en = 0.5 * (r * sum(a * a for a in v) + sum(b * b for b in B)) + p / (cfg.gamma - 1)
    U = np.stack([r * v[0], r * v[1], r * v[2], en, r, *B, f(0.0, 0.01) * np.sqrt(pr) * v0])  # psi: B times a speed
    s = Solver(cfg).put_state(U)
    g = Grid.from_solver_config(cfg, omp=True)
    g.U[...] = s.get_state_numpy()
    s.step(2)
    assert s.sync().status == 0
    g.step(2)
    unit = np.array([ro * v0] * 3 + [pr, ro] + [np.sqrt(pr)] * 3 + [np.sqrt(pr) * v0]).reshape((9,) + (1,) * nd)
    assert_parity(s.get_state_numpy() / unit, g.U / unit, 1e-12, f"rho {ro} p {pr}")
