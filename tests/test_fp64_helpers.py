"""The kernels' FP64 reciprocal and grid position, on the device, against their
exact values, and the plain sum where its reciprocal hands over to a division.
"""
import numpy as np
import pytest

import hkb
from hkb import synth

pytestmark = pytest.mark.gpu


def test_reciprocal():
    """Every exponent from the smallest normal number to 1e300, random mantissas
    and those at both ends of a binade.  The start keeps the upper word's 20 bits
    of mantissa in its argument and its result, 2^-19 together; the step leaves
    their cube, 2^-57, beside the last rounding's 2^-53.  Bound: 1.25 x 2^-53."""
    rng = np.random.default_rng(1)
    e = np.arange(-1022, 997)
    m = np.concatenate([1.0 + rng.random(500), [1.0, np.nextafter(1.0, 2.0), 1.5, np.nextafter(2.0, 1.0),
                                                1.0 + 2.0 ** -20, 1.0 + 2.0 ** -21, 1.0 + 2.0 ** -52]])
    v = np.ldexp(m[None, :], e[:, None]).ravel()
    v = v[v <= 1e300]
    with hkb.Context(0) as ctx:
        got = ctx.fp64_eval(0, v)
    err = np.abs(np.longdouble(1.0) - got.astype(np.longdouble) * v.astype(np.longdouble))
    # (the product of two 53-bit numbers in 64 bits: half a unit of 2^-63 more)
    print(f"reciprocal: at most {float(err.max()) * 2.0 ** 53:.4f} x 2^-53")
    assert err.max() <= 1.25 * 2.0 ** -53
    div = 1.0 / v
    assert (np.abs(got - div) <= np.spacing(div)).all()


def test_grid_position():
    """2 j / den - 1 as the division gives it: whole grids, odd and even, and random pairs."""
    rng = np.random.default_rng(2)
    j, den = [], []
    for d in (1, 2, 3, 4, 7, 119, 120, 1023, 3071, 3072, 9998, 9999, 10000, 12287, 12288):
        j.append(np.arange(d + 1))
        den.append(np.full(d + 1, d))
    d = rng.integers(12300, 2 ** 31 - 1, 1_000_000)
    j.append(np.floor(d * rng.random(len(d))))
    den.append(d)
    j, den = np.concatenate(j).astype(np.float64), np.concatenate(den).astype(np.float64)
    with hkb.Context(0) as ctx:
        assert np.array_equal(ctx.fp64_eval(1, j, den), 2.0 * j / den - 1.0)
        for bad in ((-1.0, 4.0), (5.0, 4.0), (0.5, 4.0), (0.0, 0.0), (1.0, 2.0 ** 31)):
            with pytest.raises(hkb.HkError) as e:
                ctx.fp64_eval(1, [bad[0]], [bad[1]])
            assert e.value.status == -1
        with pytest.raises(hkb.HkError):
            ctx.fp64_eval(2, [1.0])


@pytest.mark.parametrize("mass", [1.0, 1e290, 1e292, 1e294])
def test_plain_sum_on_both_sides_of_the_division(mass):
    """x^2 + y^2 of the tile's ends below and above 1e300, where the plain sum's
    region A goes from the reciprocal to a division: y = 0 or finite, the
    Lorentzian S y / pi / (x^2 + y^2) at 1e-14 (two roundings of x twice, of
    the reciprocal, the product and the sum)."""
    numin, dnu, nx, T, P = 1000.0, 2.0 ** -5, 2048, 600.0, 1.0
    L = synth.hitran_lines(1, seed=5, nu_min=numin + 0.4, nu_max=numin + 0.5)
    Tq, Qq = synth.q_table()
    with hkb.Context(0) as ctx:
        ctx.set_species(hkb.HITRAN, [mass * synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=1.0)
        ctx.load_lines_hitran(L)
        ctx.set_grid(numin, numin + nx * dnu, dnu, 1, 0, 1e6)
        nu, S, iad, vy, win = ctx.state_lines(T, P)
        K = ctx.opacity([T], [P], hkb.PLAIN_FP64)[0]
    x = (numin + np.arange(nx) * dnu - nu[0]) * iad[0]
    r2 = x * x + vy[0] * vy[0]
    a = r2 >= 1e6
    if mass > 1e293:
        assert r2.max() > 1e299
    want = (S[0] * vy[0] / np.pi / r2)[a]
    assert a.sum() > nx // 2
    np.testing.assert_allclose(K[a], want, rtol=1e-14)
