"""The transmission function's block sums: values with every spread against m
(one exponential and a polynomial per block, value by value, zero), block
remainders, unsorted and non-finite values, and bins too large for shared
memory, against the oracle on the same values (rtol 1e-12, as test_means.py).
"""
import numpy as np
import pytest

import hkb
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxb,nb,nTr,dTr", [(3, 2, 33, 1.0), (31, 3, 40, 2.0), (33, 2, 64, 2.0),
                                            (4097, 2, 200, 0.5), (14000, 2, 64, 1.0),
                                            (16000, 2, 64, 1.0), (40000, 1, 32, 2.0)])
@pytest.mark.parametrize("kind", ["sorted", "unsorted", "flat", "zeros"])
def test_block_sums(nxb, nb, nTr, dTr, kind):
    rng = np.random.default_rng(nxb)
    K = 10.0 ** rng.uniform(-9.0, 6.0, (nb, nxb))
    if kind == "flat":
        K = 3.0 + 1e-9 * rng.random((nb, nxb))
    elif kind == "zeros":
        K[:, : nxb // 2] = 0.0
    if kind != "unsorted":
        K = np.sort(K, axis=1)
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, nb * nxb * 0.01, 0.01, nb, 0, 25.0)
        got = ctx.transmission(K.reshape(1, -1), None, nTr, dTr)[0]
    want = oracle.transmission(K.ravel(), nxb, nb, None, 0.0, nTr, dTr)
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-290)


def test_infinite_value():
    """exp(-inf) adds nothing; the other values of the block keep theirs."""
    K = np.sort(10.0 ** np.random.default_rng(5).uniform(-3.0, 3.0, 640))
    K[-40:] = np.inf
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, 6.4, 0.01, 1, 0, 25.0)
        got = ctx.transmission(K.reshape(1, -1), None, 32, 1.0)[0]
    want = oracle.transmission(K, 640, 1, None, 0.0, 32, 1.0)
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-290)
