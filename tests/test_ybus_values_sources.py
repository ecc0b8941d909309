"""Ybus values handed over on the device: which sources and streams the plan's kernel may take directly
(another device's stream or memory, and sources that are not 16-byte aligned, go through a copy, which
takes them all), and a source 8 bytes past a 16-byte boundary against the same values aligned."""
import numpy as np
import pytest

from conftest import grid_problem


@pytest.mark.parametrize("plan,stream,source,address,route", [
    (0, 0, 0, 4096, 0), (1, 1, 1, 4096, 0),
    (0, 0, 0, 4104, 1), (0, 0, 1, 4096, 1), (0, 0, -1, 4096, 1),
    (1, 0, 1, 4096, 2), (0, 1, 0, 4096, 2), (1, 0, 0, 4104, 2)])
def test_route(plan, stream, source, address, route):
    from lightsim2grid_b200 import _native

    assert _native.load().pf_host_ybus_route(plan, stream, source, address) == route


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["newton", "dc"])
def test_source_off_a_16_byte_boundary(kind):
    import torch

    from lightsim2grid_b200 import Plan, _native as nat

    c = grid_problem("grid118")
    g = c["grid"]
    Y = (g.get_dcYbus() if kind == "dc" else c["Ybus"]).tocsc()
    Y.sort_indices()
    plan = Plan(Y, c["V0"], c["Sbus"], c["ref"], c["weights"], c["pv"], c["pq"], **({"dc": True} if kind == "dc" else {}))
    Y2 = Y.copy()
    Y2.data = 1.01 * Y.data
    plan.set_ybus_values(Y2.data)
    want = plan.solve(c["V0"], c["Sbus"], 10, 1e-8)[0]
    plan.set_ybus_values(Y.data)
    base = plan.solve(c["V0"], c["Sbus"], 10, 1e-8)[0]
    assert not np.array_equal(base, want)
    lib = plan._lib
    st = torch.cuda.current_stream().cuda_stream
    coo = Y.tocoo()
    r, cc = coo.row.astype(np.int32), coo.col.astype(np.int32)
    pos = np.zeros(r.size, np.int32)
    assert lib.pf_ybus_positions(plan.handle, int(r.size), r.ctypes.data, cc.ctypes.data, pos.ctypes.data) == 0
    stored = np.zeros(r.size, np.complex128)

    def put(data, shift):
        stored[pos] = data
        buf = torch.zeros(2 * r.size + 2, dtype=torch.float64, device="cuda")
        buf[shift:shift + 2 * r.size] = torch.from_numpy(stored.view(np.float64)).cuda()
        nat.check(lib.pf_set_ybus_values_device(plan.handle, buf.data_ptr() + 8 * shift, st),
                  "pf_set_ybus_values_device", lib)
        torch.cuda.synchronize()

    for shift in (0, 1):
        put(Y.data, 0)
        assert np.array_equal(plan.solve(c["V0"], c["Sbus"], 10, 1e-8)[0], base)
        put(Y2.data, shift)
        assert np.array_equal(plan.solve(c["V0"], c["Sbus"], 10, 1e-8)[0], want), shift
