"""Substitution programs of the fast decoupled kernel as padded rows: systems of one to a few hundred
unknowns (row counts around the 32-row masks and the 4 rows loaded ahead) and every thread count,
against the oracle at the bars of the other fast decoupled tests (same iterations and error codes,
|dV| <= 1e-9); no PQ bus leaves the second system empty."""
import numpy as np
import pytest

from oracle.fdpf import fdpf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [0, 32, 96, 256])
@pytest.mark.parametrize("n,npv", [(3, 1), (5, 1), (14, 4), (14, 13), (33, 5), (64, 40), (150, 20), (300, 60)])
def test_sizes(n, npv, threads):
    from lightsim2grid_b200 import Plan, synthetic

    g, V = synthetic.make_grid(n, max(n - 1, int(1.3 * n)) if n > 5 else n, npv, seed=n)
    Y = g.get_Ybus()
    S = 0.98 * V * np.conj(Y @ V)
    a = (g.get_slack_ids(), g.get_slack_weights(), g.get_pv(), g.get_pq())
    Bp, Bpp = g.get_Bp_Bpp(1)
    Vo, conv_o, it_o, err_o = fdpf(Y, V, S, *a, Bp, Bpp, 40, 1e-8)
    plan = Plan(Y, V, S, *a, fdpf=(Bp, Bpp), threads=threads)
    for _ in range(2):
        Vg, conv, it, err = plan.solve(V, S, 40, 1e-8)
        assert (conv, it, err) == (conv_o, it_o, err_o)
        assert np.abs(Vg - Vo).max() <= 1e-9
