"""Error of the fit's reconstruction against its series in extended precision
(numpy longdouble), for the coefficients that the same call returns.

Tolerance on the root mean square of the relative error: 1.2e-15.  exp turns the
absolute error of f = ln K into a relative one.  |f| lies below 16 at nearly all
points, where a rounding is uniform in a spacing of at most 2^-49 (0.5e-15 rms):
two such for the large terms and their sum, 0.7e-15, and 0.2e-15 each for exp,
the scale and the product give 0.8e-15; half as much again for the small terms.
"""
import numpy as np
import pytest

import hkb
from test_fit_accuracy import spectra

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxb,nC", [(24, 4), (25, 5), (119, 20), (600, 100), (1500, 1), (1500, 2), (1500, 3), (1501, 8),
                                    (3000, 25), (10000, 20), (12288, 30)])
def test_reconstruction(nxb, nC):
    nb, LD = 6, np.longdouble
    K = spectra(nb, nxb, nxb)
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, nb * nxb * 0.01, 0.01, nb, 0, 25.0)
        r = ctx.kdist(K.reshape(1, -1), nC=nC, recon=True)
    x = -1 + np.arange(nxb).astype(LD) * 2 / LD(nxb)
    T = [np.ones_like(x), x]
    for i in range(2, nC):
        T.append(2 * x * T[-1] - T[-2])
    want = np.exp(r["coeff"][0].astype(LD) @ np.array(T[:nC]))
    err = (np.abs(r["recon"][0].reshape(nb, nxb) - want) / want).astype(np.float64)
    print(nxb, nC, f"reconstruction: rms {np.sqrt((err ** 2).mean()):.2e}, max {err.max():.2e}")
    assert np.sqrt((err ** 2).mean()) < 1.2e-15
