"""The transmission function where its kernel chooses between a block's power
sums and its single values: bins and orders below and above the sizes at which
power sums are formed, unsorted values whose blocks are too wide for every,
all but one, two or three of the m_j, m_j descending and constant, and groups of
blocks that are summed whole, against the oracle (rtol 1e-12, as
test_transmission_blocks.py).
"""
import numpy as np
import pytest

import hkb
import oracle

pytestmark = pytest.mark.gpu


def check(K, nxb, nb, nTr, dTr):
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, nb * nxb * 0.01, 0.01, nb, 0, 25.0)
        got = ctx.transmission(K.reshape(1, -1), None, nTr, dTr)[0]
    want = oracle.transmission(K.ravel(), nxb, nb, None, 0.0, nTr, dTr)
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-290)


@pytest.mark.parametrize("nxb,nb,nTr", [(511, 2, 60), (512, 2, 58), (512, 2, 59), (1000, 3, 29), (1000, 3, 31),
                                        (1024, 2, 200), (1025, 2, 200), (10007, 1, 3), (10007, 1, 64)])
@pytest.mark.parametrize("dTr", [0.05, 0.7, -0.7, 0.0])
@pytest.mark.parametrize("sort", [False, True])
def test_sizes(nxb, nb, nTr, dTr, sort):
    K = 10.0 ** np.random.default_rng(nxb + nTr).uniform(-8.0, 5.0, (nb, nxb))
    check(np.sort(K, axis=1) if sort else K, nxb, nb, nTr, dTr)


@pytest.mark.parametrize("few", [0.5, 1.5, 2.5, 3.5])
def test_blocks_that_serve_few_m(few):
    """Spread times the smallest, second, third, fourth m_j just below 1."""
    nxb, nTr, dTr = 2048, 40, 1.0
    m = np.exp((np.arange(nTr) - nTr // 2) * dTr)
    h = 1.0 / (m[0] * np.exp(few * dTr))
    K = h * 2.0 * np.random.default_rng(3).random((1, nxb))
    check(K, nxb, 1, nTr, dTr)
