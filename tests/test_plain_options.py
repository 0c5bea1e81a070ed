"""The plain form's option kernels (profiles 2-4, sub-Lorentzian wings, plinth
removal): a small state, whose tiles are split into sub-tiles, has the bits of
the same state in a batch of whole tiles and in both table modes, and meets
the oracle (1e-12; with plinth removal 1e-9, as test_profiles.py).
"""
import numpy as np
import pytest

import hkb
import oracle
from hkb import synth

pytestmark = pytest.mark.gpu

SL14 = [3.0, 10.0, 20.0, 0.09, -0.05, 0.004, 0.05, 0.02, 0.003, 0.02, 0.0, 0.0, 1000.0, 1100.0]


@pytest.mark.parametrize("nx,n", [(50, 1), (2049, 100), (10000, 3000)])
@pytest.mark.parametrize("profile,plinth,sub", [(2, 0, 0), (3, 0, 0), (4, 0, 0), (1, 1, 0), (2, 1, 0), (1, 0, 1),
                                                (1, 1, 1)])
def test_small_state(nx, n, profile, plinth, sub):
    import torch
    numin, dnu, cut, T, P = 1000.0, 0.01, 25.0, 700.0, 0.4
    L = synth.hitran_lines(n, seed=nx + n, nu_min=numin - 5.0, nu_max=numin + nx * dnu + 5.0)
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
        K = ctx.opacity([T], [P], hkb.PLAIN_FP64)[0]
        Kb = ctx.opacity([T] * 300, [P] * 300, hkb.PLAIN_FP64)
        Kt = torch.empty(5, nx, dtype=torch.float64, device="cuda")
        co = torch.empty(5, 1, 4, dtype=torch.float64, device="cuda")
        nm = torch.empty(5, 1, dtype=torch.int32, device="cuda")
        for mode in (0, 1):
            ctx.set_table_mode(mode)
            ctx.table_build([T] * 5, [P] * 5, Kt, co, nm, nC=4, precision=hkb.PLAIN_FP64)
            ctx.table_run()
            ctx.table_status()
            assert np.array_equal(Kt.cpu().numpy(), np.broadcast_to(K, (5, nx)))
        ctx.table_free()
    assert np.array_equal(Kb, np.broadcast_to(K, Kb.shape))
    if sub:
        return  # its values: test_profiles.py
    Q = oracle.partition(Tq, Qq, T)
    nu, S, iad, vy = oracle.prep_hitran(L, [synth.MASS], [1.0], [Q], T, P, qalphaL=1.0)
    win = oracle.windows(nu, S, iad, vy, numin, dnu, nx, 0, cut, profile=profile)
    pl = oracle.plinth(S, iad, vy, win, 0, cut, profile) if plinth else None
    Kref, _ = oracle.opacity(nu, S, iad, vy, win, numin, dnu, nx, profile=profile, plinth=pl)
    m = np.abs(Kref) > 1e-6 * np.abs(Kref).max()
    # (a Doppler line may reach none of 50 points)
    assert (np.abs(K - Kref)[m] / np.abs(Kref)[m]).max(initial=0.0) < (1e-9 if plinth else 1e-12)
