"""Sort of bins in which some values crowd into one step of the distribution
sort: crowds that the first look at every thread's first value finds, that only
the full count finds, and at the edge of the longest run sorted in place.
Sorted values bit-exact.
"""
import numpy as np
import pytest

import hkb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxb", [2000, 5000, 10000])
@pytest.mark.parametrize("crowd", [1, 63, 64, 65, 66, 100, 700, 1900])
@pytest.mark.parametrize("first", [False, True])
def test_crowd(nxb, crowd, first):
    rng = np.random.default_rng(nxb + crowd)
    K = 10.0 ** rng.uniform(-8.0, 5.0, (3, nxb))
    for b in range(3):
        # neighbours in the order of the bit patterns: one step
        at = np.arange(crowd) if first else rng.choice(nxb, crowd, replace=False)
        K[b, at] = np.nextafter(1.5, 2.0) + rng.integers(0, crowd, crowd) * 2.0 ** -50
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, 3 * nxb * 0.01, 0.01, 3, 0, 25.0)
        got = ctx.kdist(K.reshape(1, -1), coeff=False, nxmin=False, sorted_K=True)["sorted"][0]
    assert np.array_equal(got.reshape(3, nxb), np.sort(K, axis=1))
