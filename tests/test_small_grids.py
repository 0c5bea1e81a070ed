"""Small calls: a state whose tiles are split into sub-tiles and many parts of
their line range gives the same K, bit for bit, as the same state inside a
batch large enough for whole tiles, and meets the FP64 oracle.

Tolerances as in test_gpu_parity.py: plain 1e-12, mixed 1e-5 relative where K
exceeds 1e-6 of its maximum.
"""
import numpy as np
import pytest

import hkb
import oracle
from hkb import synth

pytestmark = pytest.mark.gpu


# points (below one 64-point block, one tile and a point, ragged, several
# tiles) x lines (one, below a chunk, one chunk a part, several)
@pytest.mark.parametrize("nx,n", [(50, 1), (50, 3000), (2049, 100), (4111, 5000), (10000, 2000),
                                  (20000, 9000)])
@pytest.mark.parametrize("precision", [hkb.MIXED, hkb.PLAIN_FP64])
def test_small_state_equals_batch_and_oracle(nx, n, precision):
    numin, dnu, cut, T, P = 1000.0, 0.01, 25.0, 700.0, 0.4
    L = synth.hitran_lines(n, seed=nx + n, nu_min=numin - 20.0, nu_max=numin + nx * dnu + 20.0)
    Tq, Qq = synth.q_table()
    with hkb.Context(0) as ctx:
        ctx.set_species(hkb.HITRAN, [synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=1.0)
        ctx.load_lines_hitran(L)
        ctx.set_grid(numin, numin + nx * dnu, dnu, 1, 0, cut)
        K = ctx.opacity([T], [P], precision)[0]
        # 700 copies: more tickets than any rule turns into sub-tiles
        Kb = ctx.opacity([T] * 700, [P] * 700, precision)
    assert np.array_equal(K, Kb[0]) and np.array_equal(K, Kb[-1])
    Q = oracle.partition(Tq, Qq, T)
    nu, S, iad, vy = oracle.prep_hitran(L, [synth.MASS], [1.0], [Q], T, P, qalphaL=1.0)
    win = oracle.windows(nu, S, iad, vy, numin, dnu, nx, 0, cut)
    Kref, _ = oracle.opacity(nu, S, iad, vy, win, numin, dnu, nx)
    m = Kref > 1e-6 * Kref.max()
    err = np.abs(K - Kref)[m] / Kref[m]
    assert err.max() < (1e-12 if precision == hkb.PLAIN_FP64 else 1e-5)
