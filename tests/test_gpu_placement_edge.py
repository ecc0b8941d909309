"""A plan whose shared-memory LU leaves 2,204 bytes of a CTA's shared memory: it is taken (2,048 bytes are kept
for the kernels' static part) and runs in batch launches and in the request loop, whose kernel has the
largest static part, with the same results, equal to the oracle's."""
import numpy as np
import pytest

from oracle.oracle import OracleNR

pytestmark = pytest.mark.gpu


def test_largest_shared_memory_plan_runs_in_every_kernel():
    import torch

    from lightsim2grid_b200 import synthetic
    from lightsim2grid_b200.serving import N1, PF, PowerFlowServer, Request

    g, _ = synthetic.make_grid(1504, 1955, 250, seed=1504)
    args = (g.get_slack_ids(), g.get_slack_weights(), g.get_pv(), g.get_pq())
    srv = PowerFlowServer({"g": g}, precision=0, slots=4, device_loop=True, lu_placement=1, threads=768)
    sv = srv.services["g"]
    left = torch.cuda.get_device_properties(0).shared_memory_per_block_optin - sv.plan.info()["shared_bytes"]
    assert sv.plan.info()["lu_in_shared"] == 1 and 2048 <= left < 2320
    reqs = [Request(k, "g", PF, 0.0, scale=np.full(g.n_bus, 1.0 - 0.02 * k)) for k in range(3)]
    reqs.append(Request(3, "g", N1, 0.0, branches=np.arange(0, 40, 5)))
    done = {r.rid: r for r in srv.serve(reqs, realtime=False)}
    assert len(done) == 4
    for k in range(3):
        o = OracleNR(False)
        assert o.compute_pf(g.get_Ybus(), sv.Vbase, sv.Sbase * (1.0 - 0.02 * k), *args, 10, 1e-8)
        assert done[k].converged[0] and np.abs(done[k].V[0] - o.get_V()).max() <= 1e-10
    V, conv, it, err = sv.plan.batch_n1([g.branch_coeffs([b]) for b in range(0, 40, 5)], sv.Vbase, sv.Sbase, 10, 1e-8)
    assert np.array_equal(done[3].converged, conv) and np.array_equal(done[3].V[conv], V[conv]) and conv.any()
