"""Branch flows on both sides of the row size where the launch shape changes, with zero, tiny, infinite and
NaN voltages and several removed branches per row: |I_ft| sn / (sqrt(3) vn) and Re(S_ft) sn in numpy,
NaN amps where the reference's quotient |E_f I_ft| / |E_f| has none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 14, 1499, 1500, 3000])
@pytest.mark.parametrize("rows", [1, 7, 700])
def test_edges(n, rows):
    from lightsim2grid_b200 import synthetic
    from lightsim2grid_b200.flows import BranchSet, flows_host

    g, V0 = synthetic.make_grid(n, max(n - 1, int(1.2 * n)) if n > 5 else n - 1, max(1, n // 8), seed=n)
    rng = np.random.default_rng(n + rows)
    V = V0[None, :] * (1.0 + 0.02 * rng.standard_normal((rows, n))) * np.exp(1j * rng.uniform(-3, 3, (rows, n)))
    V[0] = 0.0
    if rows > 4:
        V[1, ::3] = 0.0
        V[2, ::2] *= 1e-140
        V[3, 0] = np.nan
        V[4, 1] = np.inf
    br = BranchSet(g)
    br.status[::5] = 0
    removed = [rng.choice(br.nbr, size=min(br.nbr, k % 4), replace=False).tolist() for k in range(rows)]
    a, p = flows_host(br, V, removed=removed)
    with np.errstate(all="ignore"):
        ef, et = V[:, br.from_], V[:, br.to]
        I = np.conj(br.yff * ef + br.yft * et)
        ar = np.abs(I) * br.sn_mva / (np.sqrt(3.0) * br.vn_kv_from)
        ar[~((np.abs(ef) > 0) & np.isfinite(ef))] = np.nan
        pr = (ef.real * I.real - ef.imag * I.imag) * br.sn_mva
        scale = (np.abs(br.yff) * np.abs(ef) + np.abs(br.yft) * np.abs(et)) * br.sn_mva
    # no rounding is allowed where a term is not finite: such values are exact zeros (removed branches)
    scale[~np.isfinite(scale)] = 0.0
    ef = np.where(np.isfinite(ef), ef, 0.0)
    ar[:, br.status == 0] = pr[:, br.status == 0] = 0.0
    for k, lst in enumerate(removed):
        for b in lst:
            ar[k, b] = 0.0 if np.isfinite(ar[k, b]) else ar[k, b]
            pr[k, b] = 0.0 if np.isfinite(pr[k, b]) else pr[k, b]
    assert np.array_equal(np.isnan(a), np.isnan(ar))
    assert np.array_equal(np.isfinite(p), np.isfinite(pr))
    ok = np.isfinite(ar)
    # the two terms of I cancel: a few roundings of their sizes
    assert np.all(np.abs(a - ar)[ok] <= 8e-16 * (scale / (np.sqrt(3.0) * br.vn_kv_from))[ok] + 1e-15 * ar[ok] + 1e-300)
    ok = np.isfinite(pr)
    assert np.all(np.abs(p - pr)[ok] <= 8e-16 * (scale * np.abs(ef))[ok] + 1e-300)
