"""Tickets without work: a tile with fewer chunks of lines than parts of its
line range, or with no line, ends its ticket without a block barrier, and
the CTA's warps still have to take the next ticket together.

A few lines at one end of a grid of several tiles, many states in one launch:
most tickets return at once.  Every state's row has the bits of the same
state alone, in each form of the sum (mixed Voigt, plain FP64, Doppler,
sub-Lorentzian wings, plinth removal), and the Voigt rows meet the oracle at
the tolerances of test_gpu_parity.py.
"""
import numpy as np
import pytest

import hkb
import oracle
from hkb import synth

pytestmark = pytest.mark.gpu

SL14 = [3.0, 10.0, 20.0, 0.09, -0.05, 0.004, 0.05, 0.02, 0.003, 0.02, 0.0, 0.0, 1000.0, 1100.0]


@pytest.mark.parametrize("n", [1, 300])
@pytest.mark.parametrize("profile,plinth,sub,precision", [(1, 0, 0, hkb.MIXED), (1, 0, 0, hkb.PLAIN_FP64),
                                                          (3, 0, 0, hkb.MIXED), (1, 0, 1, hkb.MIXED),
                                                          (1, 1, 0, hkb.MIXED), (2, 0, 0, hkb.MIXED)])
def test_tickets_without_work(n, profile, plinth, sub, precision):
    numin, dnu, nx, cut, T, P = 1000.0, 0.01, 9000, 5.0, 900.0, 0.3
    L = synth.hitran_lines(n, seed=n, nu_min=numin + 1.0, nu_max=numin + 4.0)
    Tq, Qq = synth.q_table()
    with hkb.Context(0) as ctx:
        ctx.set_species(hkb.HITRAN, [synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=1.0)
        ctx.load_lines_hitran(L)
        ctx.set_grid(numin, numin + nx * dnu, dnu, 1, 0, cut)
        ctx.set_profile(profile, plinth)
        if sub:
            ctx.set_sublorentzian(SL14)
        one = ctx.opacity([T], [P], precision)[0]
        many = [ctx.opacity([T] * 400, [P] * 400, precision) for _ in range(3)]
    for K in many:
        assert np.array_equal(K, np.broadcast_to(one, K.shape))
    if profile == 1 and not plinth and not sub:
        Q = oracle.partition(Tq, Qq, T)
        nu, S, iad, vy = oracle.prep_hitran(L, [synth.MASS], [1.0], [Q], T, P, qalphaL=1.0)
        win = oracle.windows(nu, S, iad, vy, numin, dnu, nx, 0, cut)
        Kref, _ = oracle.opacity(nu, S, iad, vy, win, numin, dnu, nx)
        m = Kref > 1e-6 * Kref.max()
        err = np.abs(one - Kref)[m] / Kref[m]
        assert err.max() < (1e-12 if precision == hkb.PLAIN_FP64 else 1e-5)
