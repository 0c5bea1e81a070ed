"""The per-bin sort and fit at the sizes and values where its kernels change:
edges of the CTA and keys-per-thread classes, the shared-memory limit, bins
whose values crowd, tie, sit at the floor or are not finite.

Sorted values bit-exact; coefficients 1e-9 absolute against the oracle on the
same K (as test_gpu_parity.py).
"""
import numpy as np
import pytest

import hkb
import oracle

pytestmark = pytest.mark.gpu


def spectra(kind, nb, nxb, seed):
    rng = np.random.default_rng(seed)
    K = 10.0 ** rng.uniform(-8.0, 5.0, (nb, nxb))
    if kind == "crowded":     # all but a few values within 1e-4: too many per step
        K = 1.0 + 1e-4 * rng.random((nb, nxb))
        K[:, ::97] = 1e9
    elif kind == "ties":      # few distinct values
        K = 10.0 ** rng.integers(-3, 4, (nb, nxb)).astype(np.float64)
    elif kind == "floor":     # points without lines
        K[rng.random((nb, nxb)) < 0.4] = 0.0
        K[0] = 0.0
    return K


def fit(K, nC):
    nb, nxb = K.shape
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, nb * nxb * 0.01, 0.01, nb, 0, 25.0)
        return ctx.kdist(K.reshape(1, -1), nC=nC, sorted_K=True)


@pytest.mark.parametrize("nxb,nb,nC", [(4, 3, 4), (24, 5, 4), (120, 3, 20), (119, 3, 20), (1024, 150, 8),
                                       (1025, 300, 20), (2049, 300, 12), (3072, 300, 30), (3073, 150, 20),
                                       (6145, 2, 100), (10000, 3, 20), (12288, 2, 21), (12289, 2, 20)])
@pytest.mark.parametrize("kind", ["spread", "crowded", "ties", "floor"])
def test_sizes(nxb, nb, nC, kind):
    K = spectra(kind, nb, nxb, nxb + nC)
    r = fit(K, nC)
    Ks = np.sort(K, axis=1)
    assert np.array_equal(r["sorted"][0].reshape(nb, nxb), Ks)
    with np.errstate(divide="ignore", invalid="ignore"):
        co, nxmin, _ = oracle.kdist(Ks.ravel(), nxb, nb, nC)
    assert np.array_equal(r["nxmin"][0], nxmin)
    got = r["coeff"][0]
    assert np.array_equal(np.isfinite(got), np.isfinite(co))
    m = np.isfinite(co)
    assert np.abs(got - co)[m].max(initial=0.0) < 1e-9


@pytest.mark.parametrize("nxb,nC", [(600, 6), (10000, 20)])
def test_non_finite_value(nxb, nC):
    """A bin with an infinite value has no finite coefficient; the others keep theirs."""
    K = spectra("spread", 3, nxb, 1)
    ref = fit(K, nC)["coeff"][0]
    K[1, nxb // 3] = np.inf
    r = fit(K, nC)
    assert np.array_equal(r["sorted"][0].reshape(3, nxb), np.sort(K, axis=1))
    got = r["coeff"][0]
    assert np.isnan(got[1]).all() and np.array_equal(got[[0, 2]], ref[[0, 2]])
