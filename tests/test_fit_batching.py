"""A state's coefficients, sorted values and reconstruction have the same bits
whether it is fitted alone or in a batch of any size, and in a table as by
opacity + kdist of each state: bin sizes of every CTA width of the fit, by
moments and by reflections, with batches on both sides of one CTA per SM.
"""
import numpy as np
import pytest

import hkb
from hkb import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxb,nb,nC", [(60, 20, 20), (500, 20, 3), (1000, 20, 20), (3000, 20, 30), (3073, 10, 20),
                                       (5000, 20, 20), (9000, 12, 20), (12289, 2, 20)])
def test_state_alone_equals_state_in_batch(nxb, nb, nC):
    ns = 24
    K = 10.0 ** np.random.default_rng(nxb).uniform(-8.0, 5.0, (ns, nb * nxb))
    K[:, 5:9] = 0.0
    with hkb.Context(0) as ctx:
        ctx.set_grid(0.0, nb * nxb * 0.01, 0.01, nb, 0, 25.0)
        batch = ctx.kdist(K, nC=nC, sorted_K=True, recon=True)
        for s in (0, 7, ns - 1):
            one = ctx.kdist(K[s:s + 1], nC=nC, sorted_K=True, recon=True)
            for key in ("coeff", "nxmin", "sorted", "recon"):
                assert np.array_equal(one[key][0], batch[key][s], equal_nan=True), key


def test_table_equals_states_one_by_one():
    import torch
    nb, nxb = 40, 1000
    L = synth.hitran_lines(3000, seed=3, nu_min=500.0, nu_max=900.0)
    Tq, Qq = synth.q_table()
    T, P = np.linspace(300.0, 2000.0, 12), np.full(12, 0.2)
    with hkb.Context(0) as ctx:
        ctx.set_species(hkb.HITRAN, [synth.MASS], [1.0])
        ctx.set_partition(0, Tq, Qq)
        ctx.set_options(qalphaL=1.0)
        ctx.load_lines_hitran(L)
        ctx.set_grid(500.0, 900.0, 0.01, nb, 0, 25.0)
        K = torch.empty(12, nb * nxb, dtype=torch.float64, device="cuda")
        co = torch.empty(12, nb, 20, dtype=torch.float64, device="cuda")
        nm = torch.empty(12, nb, dtype=torch.int32, device="cuda")
        ctx.table_build(T, P, K, co, nm)
        ctx.table_run()
        torch.cuda.synchronize()
        K, co = K.cpu().numpy(), co.cpu().numpy()
        ctx.table_free()
        for s in range(12):
            Ks = ctx.opacity(T[s:s + 1], P[s:s + 1])
            assert np.array_equal(Ks[0], K[s])
            assert np.array_equal(ctx.kdist(Ks)["coeff"][0], co[s])
