"""Zero start voltages: dS/dVa of such a bus is zero and dS/d|V| undefined, so a PV bus, which has no
magnitude unknown, leaves the Jacobian singular: SolverReFactor (6) in the first step, with the start
voltages as the result, as the reference ends at its factorisation.  A slack bus has neither unknown, and
its zero voltage is a start point like any other.  The Jacobian itself against dense numpy values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(n):
    from lightsim2grid_b200 import synthetic

    g, V = synthetic.make_grid(n, int(1.6 * n), max(2, n // 6), seed=n)
    return g, V, V * np.conj(g.get_Ybus() @ V)


def _args(g):
    return g.get_slack_ids(), g.get_slack_weights(), g.get_pv(), g.get_pq()


@pytest.mark.parametrize("value", [0.0, -0.0])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [14, 33, 97])
def test_pv_bus_is_a_singular_jacobian(n, precision, value):
    from lightsim2grid_b200 import Plan

    g, V, S = _grid(n)
    for distributed in (False, True):
        for bus in g.get_pv()[:3]:
            V0 = V.copy()
            V0[bus] = value
            for layout in (1, 2):
                plan = Plan(g.get_Ybus(), V, S, *_args(g), precision=precision, batch_layout=layout,
                            distributed=distributed)
                _, conv, it, err = plan.batch_n1([[]] * 3, V0, S, 10, 1e-8)
                assert not conv.any() and np.all(err == 6) and np.all(it == 1), (bus, layout)
            Vo, conv, it, err = plan.solve(V0, S, 10, 1e-8)
            assert not conv and err == 6 and it == 1 and np.array_equal(Vo, V0)


@pytest.mark.parametrize("n", [14, 33])
def test_magnitude_columns_alone_are_undefined(n):
    from lightsim2grid_b200 import Plan

    g, V, S = _grid(n)
    plan = Plan(g.get_Ybus(), V, S, *_args(g), distributed=False)
    ref, pv, pq = g.get_slack_ids(), np.asarray(g.get_pv()), np.asarray(g.get_pq())
    pvpq = np.r_[pv, pq]
    for bus in (pv[0], pq[0]):
        V0 = V.copy()
        V0[bus] = 0.0
        plan.solve(V0, S, 1, 1e-8)
        J = plan.get_J().toarray()
        Y = g.get_Ybus().toarray()
        dVa = 1j * np.diag(V0) @ np.conj(np.diag(Y @ V0) - Y @ np.diag(V0))
        want = np.r_[dVa.real[np.ix_(pvpq, pvpq)], dVa.imag[np.ix_(pq, pvpq)]]
        assert np.all(np.isfinite(J[:, :pvpq.size]))
        assert np.abs(J[:, :pvpq.size] - want).max() <= 1e-10
        bad = ~np.isfinite(J[:, pvpq.size:]).all(axis=0)
        assert np.array_equal(bad, pq == bus)
