"""Plinth removal: whole slices of one region (two points to an instruction) and
slices that a window edge or the grid's end cuts (point by point) give the
same bits.

The same lines on two grids that share every point of the shorter one: in its
last tile the points lie in slices cut by the grid's end.  One chunk of lines
of one strength level, so the order of the sums is the same.
"""
import numpy as np
import pytest

import hkb
from hkb import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [2048 + 1000, 2048 + 37, 1500, 2048 + 256, 4095])
@pytest.mark.parametrize("profile,cut,dnu", [(1, 25.0, 1e-3), (1, 25.0, 1e-2), (1, 1.5, 1e-3), (2, 25.0, 1e-2),
                                             (2, 1.5, 1e-3)])
def test_packed_equals_per_point(nx, profile, cut, dnu):
    numin, nfull, T, P = 1000.0, 4096, 900.0, 0.1
    span = nfull * dnu
    L = synth.hitran_lines(90, seed=8, nu_min=numin - 0.5 * span, nu_max=numin + 1.5 * span)
    rng = np.random.default_rng(4)
    L["S"] = np.asarray(L["S"]) * 0.0 + 10.0 ** rng.uniform(-22.0, -20.0, 90)
    L["EL"] = np.asarray(L["EL"]) * 0.0 + 100.0
    Tq, Qq = synth.q_table()
    K = []
    with hkb.Context(0) as ctx:
        ctx.set_species(hkb.HITRAN, [synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=1.0)
        ctx.load_lines_hitran(L)
        for n in (nfull, nx):
            ctx.set_grid(numin, numin + n * dnu, dnu, 1, 0, cut)
            assert ctx.nx == n
            ctx.set_profile(profile, 1)
            K.append(ctx.opacity([T], [P], hkb.MIXED)[0])
    assert (K[0] != 0.0).all()
    assert np.array_equal(K[0][:nx], K[1])
