"""The adjoint's split of a tile's lines at the ends of its rule: no line or one
line a part, parts of a few lines, one tile and several, a cutoff in Lorentz
widths (whose windows the rule does not know).  Gradients against the oracle
with the tolerances of test_adjoint.py.
"""
import numpy as np
import pytest

import hkb
import oracle
from hkb import synth

pytestmark = pytest.mark.gpu

NUMIN, DNU, T, P = 1000.0, 0.01, 800.3, 1.0


@pytest.mark.parametrize("nx,n", [(500, 1), (2049, 7), (8192, 9), (8193, 100), (3000, 6000), (40000, 3000)])
@pytest.mark.parametrize("precision,tol,tol_line", [(hkb.PLAIN_FP64, 1e-9, 1e-9), (hkb.MIXED, 1e-4, 1e-5)])
def test_parts(nx, n, precision, tol, tol_line):
    L = synth.hitran_lines(n, seed=n, nu_min=NUMIN, nu_max=NUMIN + nx * DNU)
    Tq, Qq = synth.q_table()
    with hkb.Context(0) as ctx:
        ctx.set_species(hkb.HITRAN, [synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=1.0)
        ctx.load_lines_hitran(L)
        ctx.set_grid(NUMIN, NUMIN + nx * DNU, DNU, 1, 0, 25.0)
        K = ctx.opacity([T], [P], hkb.PLAIN_FP64)[0]
        # weights of one sign: dT and dP have no cancellation between points
        u = (0.5 + np.random.default_rng(n).random(nx)) / np.maximum(K, 1e-6 * K.max())
        dT, dP, dS, dG = ctx.opacity_vjp(T, P, u, precision)
        # the same state with the cutoff in Lorentz widths, wide enough for the whole grid
        ctx.set_grid(NUMIN, NUMIN + nx * DNU, DNU, 1, 1, 1e6)
        wide = ctx.opacity_vjp(T, P, u, precision)
        ctx.set_grid(NUMIN, NUMIN + nx * DNU, DNU, 1, 0, 1e5)
        same = ctx.opacity_vjp(T, P, u, precision)
    rT, rP, rS, rG = oracle.vjp_hitran(L, synth.MASS, Tq, Qq, T, P, u, NUMIN, DNU, nx)
    assert abs(dT - rT) < tol * abs(rT) and abs(dP - rP) < tol * abs(rP)
    assert np.abs(dS - rS).max() < tol_line * np.abs(rS).max()
    assert np.abs(dG - rG).max() < tol_line * np.abs(rG).max()
    for a, b in zip(wide, same):  # every window the whole grid: the same sums
        assert np.abs(np.asarray(a) - np.asarray(b)).max() <= tol_line * np.abs(np.asarray(b)).max()
