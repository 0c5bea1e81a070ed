"""The FP64 region-C evaluator of the plain Voigt sum, and that
Context.profile_eval shows the one that runs.

Against 40-digit values at 1e-14: exp(-x^2) carries up to x^2 / 2 roundings of
its argument where it is not negligible (x < 6: 18 of 2^-53), erfcx, exp and the
sine up to four ulps, the sums a few more.
"""
import numpy as np
import pytest

import hkb
from hkb import synth

pytestmark = pytest.mark.gpu


def points():
    """The disc r < 10; tiny y; the ends of the table of denominators (nearest
    term 1 and 20), of the second sum (x near 6.4), cancelling terms; x = 0."""
    rng = np.random.default_rng(9)
    n = 400
    u = rng.random((8, n))
    r = 10.0 * np.sqrt(u[0])
    x = [r * np.cos(u[1] * np.pi / 2), 6.0 * u[2], 6.0 + 4.0 * u[3], 0.8 * u[4], 9.7 + 0.29 * u[5], 6.3 + 0.2 * u[6],
         u[7], np.zeros(8), 10.0 ** rng.uniform(-12, -1, n)]
    y = [r * np.sin(u[1] * np.pi / 2), 10.0 ** rng.uniform(-12, 0, n), 10.0 ** rng.uniform(-12, 0, n),
         10.0 ** rng.uniform(-6, 0.9, n), 10.0 ** rng.uniform(-9, -1, n), 10.0 ** rng.uniform(-6, 0.8, n),
         1.5 + u[6], 10.0 ** rng.uniform(-6, 0.9, 8), 10.0 ** rng.uniform(-3, 0.9, n)]
    x, y = np.concatenate(x), np.concatenate(y)
    m = x * x + y * y < 100.0
    return x[m], y[m]


def test_against_40_digits():
    mp = pytest.importorskip("mpmath")
    x, y = points()
    with hkb.Context(0) as ctx:
        got = ctx.profile_eval(x, y, hkb.PLAIN_FP64)
    err = np.empty(len(x))
    with mp.workdps(40):
        for i in range(len(x)):
            z = mp.mpc(x[i], y[i])
            v = mp.re(mp.exp(-z * z) * mp.erfc(mp.mpc(0, -1) * z))
            err[i] = abs((mp.mpf(got[i]) - v) / v)
    print(f"relative error: rms {np.sqrt((err ** 2).mean()):.2e}, max {err.max():.2e}")
    assert err.max() < 1e-14


@pytest.mark.parametrize("P", [1e-6, 1e-3, 0.03, 0.1, 0.3])
def test_profile_eval_is_the_sums_evaluator(P):
    """One line, points in region C only: K = Sc V(x, y) to the bit."""
    numin, dnu, nx, T = 1000.0, 2.0 ** -12, 4096, 1200.0
    L = synth.hitran_lines(1, seed=5, nu_min=numin + 0.4999, nu_max=numin + 0.5)
    Tq, Qq = synth.q_table()
    with hkb.Context(0) as ctx:
        ctx.set_species(hkb.HITRAN, [synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=1.0)
        ctx.load_lines_hitran(L)
        ctx.set_grid(numin, numin + nx * dnu, dnu, 1, 0, 25.0)
        nu, S, iad, vy, win = ctx.state_lines(T, P)
        K = ctx.opacity([T], [P], hkb.PLAIN_FP64)[0]
        c0, c1 = int(win[0, 2]), int(win[0, 3])
        assert c1 - c0 > 100
        x = (numin + np.arange(c0, c1) * dnu - nu[0]) * iad[0]   # exact grid points
        V = ctx.profile_eval(x, np.full(c1 - c0, vy[0]), hkb.PLAIN_FP64)
    assert np.array_equal(K[c0:c1], S[0] * (1.0 / 1.7724538509055160273) * V)


def test_outside_region_c():
    """Arguments beyond r = 10 are answered too (the Lorentzian's two first terms)."""
    x, y = np.array([10.5, 30.0, 0.0, 100.0]), np.array([0.1, 1.0, 12.0, 1.0])
    with hkb.Context(0) as ctx:
        got = ctx.profile_eval(x, y, hkb.PLAIN_FP64)
    z = x + 1j * y
    w = 1j / np.sqrt(np.pi) / z * (1 + 0.5 / z ** 2 + 0.75 / z ** 4 + 1.875 / z ** 6)
    np.testing.assert_allclose(got, w.real, rtol=1e-6)
