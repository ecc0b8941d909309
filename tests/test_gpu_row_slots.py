"""Ybus passes by row slots (mismatch, Jacobian fill, refinement residual) and their overrides: bus
counts around the 32-slot slices, outages whose overrides lie in up to six rows (several branches at
once), the Jacobian of a single power flow, and a zero start voltage -- against the oracle, at the bars of
the parity tests (FP64 1e-10 pu with equal iterations, mixed 1e-8 pu)."""
import numpy as np
import pytest

from oracle.oracle import OracleNR, contingency_analysis

pytestmark = pytest.mark.gpu


def _grid(n):
    from lightsim2grid_b200 import synthetic

    g, V = synthetic.make_grid(n, int(1.6 * n), max(2, n // 6), seed=n)
    return g, V, V * np.conj(g.get_Ybus() @ V)


def _args(g):
    return g.get_slack_ids(), g.get_slack_weights(), g.get_pv(), g.get_pq()


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [14, 31, 32, 33, 97, 300])
def test_outages_of_one_to_three_branches(n, precision, layout):
    from lightsim2grid_b200 import Plan

    g, V, S = _grid(n)
    rng = np.random.default_rng(n)
    lists = [rng.choice(g.nb_powerline(), size=1 + k % 3, replace=False).tolist() for k in range(24)]
    coeffs = [g.branch_coeffs(x) for x in lists]
    _, Vo, conv_o, it_o, _ = contingency_analysis(g.get_Ybus(), S, V, *_args(g), coeffs)
    plan = Plan(g.get_Ybus(), V, S, *_args(g), precision=precision, batch_layout=layout)
    Vg, conv, it, err = plan.batch_n1(coeffs, V, S, 10, 1e-8)
    assert np.array_equal(conv, conv_o) and conv.any()
    if precision == 0:
        assert np.array_equal(it[conv], it_o[conv])
    assert np.abs(Vg[conv] - Vo[conv]).max() <= (1e-10 if precision == 0 else 1e-8)


@pytest.mark.parametrize("n", [14, 33, 300])
def test_jacobian_of_the_last_step(n):
    from lightsim2grid_b200 import GPUNRSolver, GPUNRSolverSingleSlack

    g, V, S = _grid(n)
    for cls, distributed in ((GPUNRSolverSingleSlack, False), (GPUNRSolver, True)):
        o, s = OracleNR(distributed), cls()
        for x in (o, s):
            assert x.compute_pf(g.get_Ybus(), V, 1.02 * S, *_args(g), 10, 1e-8)
        assert s.get_nb_iter() == o.get_nb_iter()
        # values up to ~100 pu, a few roundings each
        assert abs(s.get_J() - o.get_J()).max() <= 1e-10


@pytest.mark.parametrize("precision", [0, 1])
def test_zero_start_voltage_is_an_infinite_value(precision):
    from lightsim2grid_b200 import Plan

    g, V, S = _grid(33)
    V0 = V.copy()
    V0[g.get_pq()[0]] = 0.0
    for layout in (1, 2):
        plan = Plan(g.get_Ybus(), V, S, *_args(g), precision=precision, batch_layout=layout)
        _, conv, it, err = plan.batch_n1([[]] * 3, V0, S, 10, 1e-8)
        assert not conv.any() and np.all(err == 3) and np.all(it == 1)
