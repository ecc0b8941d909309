"""Fast decoupled plans by the place of their factors: in global memory (padded substitution rows as wide as the
CTA, no phase tables in shared memory) at every thread count, and in shared memory (phase programs), against the
oracle at the bars of the other fast decoupled tests (same iterations and error codes, |dV| <= 1e-9); and the
256-thread form that systems above 4,000 unknowns take by default."""
import numpy as np
import pytest

from oracle.fdpf import fdpf

pytestmark = pytest.mark.gpu


def _solve(n, npv, **options):
    from lightsim2grid_b200 import Plan, synthetic

    g, V = synthetic.make_grid(n, max(n - 1, int(1.3 * n)) if n > 5 else n, npv, seed=n)
    Y = g.get_Ybus()
    S = 0.98 * V * np.conj(Y @ V)
    a = (g.get_slack_ids(), g.get_slack_weights(), g.get_pv(), g.get_pq())
    Bp, Bpp = g.get_Bp_Bpp(1)
    Vo, conv_o, it_o, err_o = fdpf(Y, V, S, *a, Bp, Bpp, 40, 1e-8)
    plan = Plan(Y, V, S, *a, fdpf=(Bp, Bpp), **options)
    for _ in range(2):
        Vg, conv, it, err = plan.solve(V, S, 40, 1e-8)
        assert (conv, it, err) == (conv_o, it_o, err_o)
        assert np.abs(Vg - Vo).max() <= 1e-9
    return plan.info()


@pytest.mark.parametrize("placement", [1, 2])
@pytest.mark.parametrize("threads", [32, 96, 128, 256, 512])
@pytest.mark.parametrize("n,npv", [(3, 1), (5, 1), (14, 13), (64, 40), (300, 60)])
def test_placements(n, npv, threads, placement):
    info = _solve(n, npv, threads=threads, lu_placement=placement)
    assert info["lu_in_shared"] == (placement == 1) and info["threads"] == threads
    if placement == 2:  # the solve vector and its padding element, rounded up to 16 bytes
        assert info["shared_bytes"] == (max(n - 1, n - 1 - npv) + 1) * 8 + 15 & ~15


def test_default_above_4000_unknowns():
    info = _solve(4200, 400)
    assert info["lu_in_shared"] == 0 and info["threads"] == 256
