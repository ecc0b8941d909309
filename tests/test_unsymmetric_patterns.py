"""LU patterns that are not symmetric -- several slack buses (the slack column and the first slack bus's row),
one-sided Ybus entries, and pivots off the diagonal at an arbitrary voltage: the elimination levels have
to follow a pivot's row as well as its column.  On the CPU the schedules solve the oracle's Jacobian and no operation
reads a value written in its phase; on the GPU power flows and outages equal the oracle's (FP64 1e-10 pu with equal
iterations, mixed 1e-8 pu), and DC angles those of a dense solve."""
import numpy as np
import pytest
import scipy.sparse.linalg as spla
from scipy.sparse.csgraph import connected_components

from oracle.oracle import OracleNR
from test_host_plan import host_schedule_solve

KINDS = ("slacks", "one-sided", "voltage")


def _case(kind, n, seed):
    from lightsim2grid_b200 import synthetic

    rng = np.random.default_rng(1000 * n + seed)
    g, V = synthetic.make_grid(n, int(1.6 * n), max(2, n // 6), seed=n + seed)
    Y = g.get_Ybus().tocsc()
    pv, pq, ref = (np.asarray(x, np.int32) for x in (g.get_pv(), g.get_pq(), g.get_slack_ids()))
    V0 = V.copy()
    if kind == "slacks":
        k = min(pv.size - 1, 4)
        ref, pv = np.r_[ref, pv[:k]].astype(np.int32), pv[k:]
    elif kind == "one-sided":
        Y = Y.tolil()
        for _ in range(max(2, n // 8)):
            r, c = rng.integers(0, n, 2)
            if r != c and Y[r, c] == 0:
                Y[r, c] = 0.05 * complex(*rng.standard_normal(2))
        Y = Y.tocsc()
    else:
        V0 = rng.uniform(0.3, 1.5, n) * np.exp(1j * rng.uniform(-2, 2, n))
    Y.sort_indices()
    w = np.zeros(n)
    w[ref] = rng.uniform(0.2, 1.0, ref.size)
    return dict(grid=g, V=V, Ybus=Y, V0=V0, ref=ref, weights=w / w.sum(), pv=pv, pq=pq)


@pytest.mark.parametrize("seed", [0, 1, 2])
@pytest.mark.parametrize("n", [14, 33, 60, 97, 150, 300])
@pytest.mark.parametrize("kind", KINDS)
def test_schedules_solve_the_jacobian(kind, n, seed):
    c = _case(kind, n, seed)
    b = np.random.default_rng(seed).standard_normal(2 * n)
    for distributed in ((True,) if kind == "slacks" else (False, True)):
        o = OracleNR(distributed)
        o.compute_pf(c["Ybus"], c["V0"], c["V0"] * np.conj(c["Ybus"] @ c["V0"]) + 1.0, c["ref"], c["weights"], c["pv"],
                     c["pq"], 1, 1e-30)
        J = o.get_J().tocsc()
        x, _ = host_schedule_solve(c, c["V0"], b[:J.shape[0]], distributed)
        xr = spla.spsolve(J, b[:J.shape[0]])
        assert np.linalg.norm(J @ x - b[:J.shape[0]]) <= 1e-9 * np.linalg.norm(b)
        assert np.abs(x - xr).max() <= 1e-6 * max(1.0, np.abs(xr).max())


@pytest.mark.gpu
@pytest.mark.parametrize("layout,placement", [(1, 1), (1, 2), (2, 0)])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [14, 33, 97, 300])
@pytest.mark.parametrize("kind", ["slacks", "one-sided"])
def test_outages(kind, n, precision, layout, placement):
    from lightsim2grid_b200 import Plan

    c = _case(kind, n, 0)
    g, V, args = c["grid"], c["V"], (c["ref"], c["weights"], c["pv"], c["pq"])
    S = V * np.conj(c["Ybus"] @ V)
    coeffs = [g.branch_coeffs([b]) for b in range(0, g.nb_powerline(), max(1, g.nb_powerline() // 24))]
    distributed = kind == "slacks"
    plan = Plan(c["Ybus"], V, S, *args, distributed=distributed, precision=precision, batch_layout=layout,
                lu_placement=placement)
    Vg, conv, it, err = plan.batch_n1(coeffs, V, S, 10, 1e-8)
    bar = 1e-10 if precision == 0 else 1e-8
    checked = 0
    for k, rows in enumerate(coeffs):
        # an outage that leaves a part tied by one-sided entries alone has a singular Jacobian
        G = g.get_Ybus().tolil()
        for r, cc, _ in rows:
            if r != cc:
                G[r, cc] = 0
        if connected_components(G.tocsr(), directed=False)[0] > 1:
            continue
        Yk = c["Ybus"].tolil()
        for r, cc, y in rows:
            Yk[r, cc] -= y
        o = OracleNR(distributed)
        ok = o.compute_pf(Yk.tocsc(), V, S, *args, 10, 1e-8)
        assert ok and conv[k] and np.abs(Vg[k] - o.get_V()).max() <= bar
        assert precision == 1 or it[k] == o.get_nb_iter()
        checked += 1
    assert checked >= len(coeffs) // 2


@pytest.mark.gpu
@pytest.mark.parametrize("placement", [1, 2])
@pytest.mark.parametrize("n", [14, 33, 97, 300])
def test_dc(n, placement):
    from lightsim2grid_b200 import Plan

    c = _case("one-sided", n, 1)
    g, V = c["grid"], c["V"]
    Y = g.get_dcYbus().tolil()
    extra = c["Ybus"].tocoo()
    for r, cc, y in zip(extra.row, extra.col, extra.data):
        if Y[r, cc] == 0 and r != cc:
            Y[r, cc] = abs(y)
    Y = Y.tocsc()
    S = V * np.conj(g.get_Ybus() @ V)
    plan = Plan(Y, V, S, c["ref"], c["weights"], c["pv"], c["pq"], dc=True, lu_placement=placement)
    Vo, conv, it, err = plan.batch_n1([[]] * 2, V, S, 10, 1e-8)
    assert conv.all()
    keep = np.setdiff1d(np.arange(n), c["ref"])
    th = np.linalg.solve(Y.toarray().real[np.ix_(keep, keep)], S.real[keep])
    got = np.angle(Vo[1] / Vo[1][c["ref"][0]])[keep]
    assert np.abs(np.angle(np.exp(1j * (got - th)))).max() <= 1e-9
