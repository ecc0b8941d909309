"""The phase programs over an LU in global memory (operations taken a few at a time, the substitutions' LU
values loaded a phase ahead): 16-byte operations on small grids whose LU is kept out of shared memory,
packed ones on a grid whose FP64 LU does not fit it, and the dense tail's -- outages against the oracle at
the bars of the parity tests (FP64 1e-10 pu with equal iterations, mixed 1e-8 pu), DC against the
shared-memory form at 1e-12."""
import numpy as np
import pytest

from oracle.oracle import contingency_analysis

pytestmark = pytest.mark.gpu


def _grid(n, chords=0):
    from lightsim2grid_b200 import synthetic

    g, V = synthetic.make_grid(n, int(1.4 * n), max(2, n // 6), seed=n, chords=chords)
    return g, V, V * np.conj(g.get_Ybus() @ V)


def _args(g):
    return g.get_slack_ids(), g.get_slack_weights(), g.get_pv(), g.get_pq()


@pytest.mark.parametrize("threads", [0, 512])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n, chords", [(4, 0), (14, 0), (33, 0), (300, 0), (1601, 0), (2848, 300)])
def test_outages(n, chords, precision, threads):
    from lightsim2grid_b200 import Plan

    g, V, S = _grid(n, chords)
    rng = np.random.default_rng(n)
    coeffs = [g.branch_coeffs([int(b)]) for b in rng.choice(g.nb_powerline(), size=min(5, n), replace=False)]
    _, Vo, conv_o, it_o, _ = contingency_analysis(g.get_Ybus(), S, V, *_args(g), coeffs)
    plan = Plan(g.get_Ybus(), V, S, *_args(g), precision=precision, lu_placement=2, batch_layout=1, threads=threads)
    Vg, conv, it, err = plan.batch_n1(coeffs, V, S, 10, 1e-8)
    assert np.array_equal(conv, conv_o) and conv.any()
    if precision == 0:
        assert np.array_equal(it[conv], it_o[conv])
    assert np.abs(Vg[conv] - Vo[conv]).max() <= (1e-10 if precision == 0 else 1e-8)


@pytest.mark.parametrize("n", [4, 14, 300])
def test_dc(n):
    from lightsim2grid_b200 import Plan

    g, V, S = _grid(n)
    coeffs = [g.dc_branch_coeffs([b]) for b in range(min(6, g.nb_powerline()))]
    res = [Plan(g.get_dcYbus(), V, S, *_args(g), dc=True, lu_placement=p).batch_n1(coeffs, V, S, 10, 1e-8) for p in (1, 2)]
    assert np.array_equal(res[0][1], res[1][1]) and res[0][1].any()
    assert np.abs(res[0][0] - res[1][0]).max() <= 1e-12
