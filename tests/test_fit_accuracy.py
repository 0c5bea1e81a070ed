"""Error of the Chebyshev coefficients against the same fit in extended
precision (numpy longdouble): sizes inside the rule of the fit by moments, at
its edges and beyond it (reflections), few and many coefficients, odd counts.

Tolerance: four times the unit rounding of the largest |ln K| -- the device's
logarithm is good to one ulp (two such roundings), the remainder and the sum
of a fit take one each; a fit averages them over the points.
"""
import numpy as np
import pytest

import hkb

pytestmark = pytest.mark.gpu


def householder(n, nc):
    """Reflections v_j (unit leading scale), their divisors and R."""
    LD = np.longdouble
    x = np.arange(n).astype(LD) * 2 / LD(n - 1) - 1
    V = np.empty((n, nc), LD)
    V[:, 0] = 1
    if nc > 1:
        V[:, 1] = x
    for i in range(2, nc):
        V[:, i] = 2 * x * V[:, i - 1] - V[:, i - 2]
    C, D = np.empty(nc, LD), np.empty(nc, LD)
    for i in range(nc):
        s = np.sqrt((V[i:, i] ** 2).sum())
        s = -s if V[i, i] < 0 else s
        D[i] = -s
        V[i, i] += s
        C[i] = s * V[i, i]
        t = (V[i:, i:i + 1] * V[i:, i + 1:]).sum(0) / C[i]
        V[i:, i + 1:] -= V[i:, i:i + 1] * t
    return V, C, D


def exact_fit(V, C, D, b):
    """Columns of b: the first nc - 1 reflections, then the substitution with
    the reference's 64 partial sums."""
    n, nc = V.shape
    w = b.astype(np.longdouble)
    for j in range(nc - 1):
        w[j:] -= V[j:, j:j + 1] * ((V[j:, j:j + 1] * w[j:]).sum(0) / C[j])
    c = w[:nc].copy()
    c[nc - 1] /= D[nc - 1]
    for i in range(nc - 2, -1, -1):
        m = min(nc, 64)
        c[i] = (c[i] - (V[i, i + 1:m, None] * c[i + 1:m]).sum(0)) / D[i]
    return c.T


def spectra(nb, nxb, seed):
    """Log-uniform values, lines over a floor, and a narrow lognormal, in turn."""
    rng = np.random.default_rng(seed)
    K = np.empty((nb, nxb))
    k = np.arange(nxb)
    for b in range(nb):
        if b % 3 == 0:
            K[b] = 10.0 ** rng.uniform(-8.0, 5.0, nxb)
        elif b % 3 == 1:
            K[b] = 1e-8 * rng.uniform(0.5, 2.0, nxb)
            for _ in range(max(8, nxb // 60)):
                w = rng.uniform(0.5, 12.0)
                K[b] += 10.0 ** rng.uniform(-7.0, 5.0) * w / ((k - rng.integers(nxb)) ** 2 + w * w)
        else:
            K[b] = np.exp(rng.normal(-12.0, 1.0, nxb))
    return K


@pytest.mark.parametrize("nxb,nC", [(24, 4), (25, 4), (119, 20), (120, 20), (125, 20), (350, 35), (480, 80),
                                    (600, 100), (1500, 3), (2858, 100), (3001, 30), (10000, 5), (10000, 20),
                                    (12288, 30), (12289, 20)])
def test_coefficients_against_extended_precision(nxb, nC):
    nb = 6
    K = spectra(nb, nxb, nxb + nC)
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, nb * nxb * 0.01, 0.01, nb, 0, 25.0)
        got = ctx.kdist(K.reshape(1, -1), nC=nC)["coeff"][0]
    b = np.log(np.sort(K, axis=1))
    want = exact_fit(*householder(nxb, nC), b.T)
    err = np.abs(got - want).max(axis=1).astype(np.float64)
    print(nxb, nC, "error / (2^-53 max|ln K|):", err / np.abs(b).max(axis=1) * 2.0 ** 53)
    assert (err <= 4.0 * 2.0 ** -53 * np.abs(b).max(axis=1)).all()
