"""Device batches whose override lists hold positions outside the Ybus pattern (pf_ybus_positions gives -1
for such an entry): they change nothing.  Every instance carries the same outage, alone or among such
positions, and gives the bits of the outage alone; so do lists of nothing else against the base case."""
import numpy as np
import pytest

from conftest import grid_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,layout,precision", [("newton", 1, 0), ("newton", 1, 1), ("newton", 2, 0),
                                                   ("newton", 2, 1), ("dc", 0, 0), ("fdpf", 0, 0)])
def test_positions_outside_the_pattern_change_nothing(kind, layout, precision):
    import torch
    from lightsim2grid_b200 import Plan, _native as nat

    c = grid_problem("grid118")
    g = c["grid"]
    Y = g.get_dcYbus() if kind == "dc" else c["Ybus"]
    kw = {"dc": True} if kind == "dc" else ({"fdpf": g.get_Bp_Bpp(0)} if kind == "fdpf" else {})
    plan = Plan(Y, c["V0"], c["Sbus"], c["ref"], c["weights"], c["pv"], c["pq"], precision=precision,
                batch_layout=layout, **kw)
    lib = plan._lib
    coeffs = g.dc_branch_coeffs([5]) if kind == "dc" else g.branch_coeffs([5])
    rows = nat.as_i32([e[0] for e in coeffs])
    cols = nat.as_i32([e[1] for e in coeffs])
    pos = np.zeros(rows.size, np.int32)
    assert lib.pf_ybus_positions(plan.handle, int(rows.size), rows.ctypes.data, cols.ctypes.data,
                                 pos.ctypes.data) == 0
    Yc = Y.tocsr()
    vals = [Yc[r, cc] - e[2] for (r, cc), e in zip(zip(rows, cols), coeffs)]
    junk = [-1, Y.nnz, 2 ** 31 - 1, -2 ** 31]
    outage = list(zip(pos.tolist(), vals))
    lists = [outage,
             [(j, 1e3 + 0j) for j in junk] + outage,
             [e for pair in zip(outage, [(j, 1e3 + 0j) for j in junk]) for e in pair],
             [],
             [(j, 1e3 + 0j) for j in junk]]
    optr = np.r_[0, np.cumsum([len(x) for x in lists])].astype(np.int32)
    opos = np.array([p for x in lists for p, _ in x], np.int32)
    oval = np.array([v for x in lists for _, v in x], np.complex128)
    dev = torch.device("cuda:0")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    n, k = g.n_bus, len(lists)
    bufs = [t(nat.as_c128(c["V0"]).ravel().view(np.float64)), t(nat.as_c128(c["Sbus"]).ravel().view(np.float64)),
            t(optr), t(opos), t(oval.view(np.float64)), t(np.arange(k, dtype=np.int32)), t(np.ones(k, np.int32))]
    dV = torch.full((k * n * 2,), 7.0, dtype=torch.float64, device=dev)
    dit = torch.full((k,), -1, dtype=torch.int32, device=dev)
    der = torch.full((k,), -1, dtype=torch.int32, device=dev)
    b = nat.PfDeviceBatch(n_inst=k, V0=bufs[0].data_ptr(), v0_stride=0, Sbus=bufs[1].data_ptr(), sbus_stride=0,
                          ovr_ptr=bufs[2].data_ptr(), ovr_pos=bufs[3].data_ptr(), ovr_val=bufs[4].data_ptr(),
                          max_iter=40, tol=1e-8, chain=0, job_first=bufs[5].data_ptr(), job_count=bufs[6].data_ptr(),
                          njobs=k, Vout=dV.data_ptr(), iters=dit.data_ptr(), errs=der.data_ptr())
    assert lib.pf_batch_device(plan.handle, nat.ctypes.byref(b), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    V = dV.cpu().numpy().view(np.complex128).reshape(k, n)
    it, er = dit.cpu().numpy(), der.cpu().numpy()
    assert np.all(er == 0)
    for i, like in ((1, 0), (2, 0), (4, 3)):
        assert it[i] == it[like] and np.array_equal(V[i], V[like]), i
    assert not np.array_equal(V[0], V[3])
