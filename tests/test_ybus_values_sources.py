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


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1])
def test_in_a_captured_graph(shift):
    """Captured on a stream and replayed, the plan takes the values that the buffer holds then."""
    import torch

    from lightsim2grid_b200 import Plan, _native as nat

    c = grid_problem("grid118")
    Y = c["Ybus"].tocsc()
    plan = Plan(Y, c["V0"], c["Sbus"], c["ref"], c["weights"], c["pv"], c["pq"])
    coo = Y.tocoo()
    r, cc = coo.row.astype(np.int32), coo.col.astype(np.int32)
    pos = np.zeros(r.size, np.int32)
    assert plan._lib.pf_ybus_positions(plan.handle, int(r.size), r.ctypes.data, cc.ctypes.data, pos.ctypes.data) == 0
    stored = np.zeros(r.size, np.complex128)
    stored[pos] = coo.data
    base = plan.solve(c["V0"], c["Sbus"], 10, 1e-8)[0]
    values = torch.from_numpy(stored.view(np.float64)).cuda()
    buf = torch.zeros(2 * r.size + 2, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        nat.check(plan._lib.pf_set_ybus_values_device(plan.handle, buf.data_ptr() + 8 * shift,
                                                      torch.cuda.current_stream().cuda_stream),
                  "pf_set_ybus_values_device", plan._lib)
    for factor in (1.01, 1.0):
        buf[shift:shift + values.numel()] = factor * values
        graph.replay()
        torch.cuda.synchronize()
        got = plan.solve(c["V0"], c["Sbus"], 10, 1e-8)[0]
        assert np.array_equal(got, base) == (factor == 1.0)


@pytest.mark.gpu
def test_while_another_stream_captures():
    """A call on another stream neither fails nor ends the capture."""
    import torch

    from lightsim2grid_b200 import Plan, _native as nat

    c = grid_problem("grid118")
    plan = Plan(c["Ybus"], c["V0"], c["Sbus"], c["ref"], c["weights"], c["pv"], c["pq"])
    buf = torch.zeros(2 * c["Ybus"].nnz, dtype=torch.float64, device="cuda")
    x = torch.zeros(4, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = x + 1
        nat.check(plan._lib.pf_set_ybus_values_device(plan.handle, buf.data_ptr(), side.cuda_stream),
                  "pf_set_ybus_values_device", plan._lib)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, x + 1)
