"""The quotients of the LU programs and of the dense tail (csrc/pf_device_math.cuh) against IEEE division, value
by value: random operands with exponents up to +-500 (FP64) and +-40 (FP32), and divisors at the ends of the
range: infinite and huge ones give zero to within the smallest normal number, zero and subnormal ones a value that
is not finite.  A small kernel includes the header."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "pf_device_math.cuh"
template <int KIND, typename T>
__global__ void quotients(const T *a, const T *b, T *q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if constexpr (KIND == 0) q[i] = l2g::lu_div(a[i], b[i]);
    else q[i] = l2g::tail_quotient(a[i], b[i], l2g::tail_reciprocal(b[i]));
}
extern "C" int run(int kind, const void *a, const void *b, void *q, int n) {
    const int g = (n + 255) / 256;
    if (kind == 0) quotients<0, double><<<g, 256>>>((const double *)a, (const double *)b, (double *)q, n);
    else if (kind == 1) quotients<1, double><<<g, 256>>>((const double *)a, (const double *)b, (double *)q, n);
    else quotients<1, float><<<g, 256>>>((const float *)a, (const float *)b, (float *)q, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    import torch
    from lightsim2grid_b200 import build

    d = tmp_path_factory.mktemp("quotient")
    (d / "q.cu").write_text(SOURCE)
    subprocess.check_call([build._nvcc()] + build.FLAGS + ["-I", build.CSRC, "-shared", "-o", str(d / "q.so"),
                                                           str(d / "q.cu")])
    lib = ctypes.CDLL(os.path.join(str(d), "q.so"))

    def run(kind, a, b):
        dt = np.float32 if kind == 2 else np.float64
        ta, tb = (torch.from_numpy(np.ascontiguousarray(x, dt)).cuda() for x in (a, b))
        q = torch.empty_like(ta)
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        torch.cuda.synchronize()
        assert lib.run(kind, p(ta), p(tb), p(q), ta.numel()) == 0
        return q.cpu().numpy()

    return run


def _values(rng, n, span, dtype):
    m = rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n)
    return np.ldexp(m, rng.integers(-span, span, n)).astype(dtype)


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_random_operands(quotients, kind):
    rng = np.random.default_rng(kind)
    dt, span = (np.float32, 40) if kind == 2 else (np.float64, 500)
    a, b = _values(rng, 1 << 22, span, dt), _values(rng, 1 << 22, span, dt)
    q, want = quotients(kind, a, b), a / b
    assert np.array_equal(q, want)


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_divisors_at_the_ends_of_the_range(quotients, kind):
    dt = np.float32 if kind == 2 else np.float64
    f = np.finfo(dt)
    edge = dt(2) ** dt(f.maxexp - 2)  # the first divisor whose reciprocal is not normal
    big = np.array([np.inf, f.max, 1.5 * edge, np.nextafter(edge, dt(np.inf)), edge], dt)
    for num in (1.0, -3.0, 0.75, 0.0):
        for b in (big, -big):
            a = np.full(b.size, num, dt)
            q, want = quotients(kind, a, b), a / b
            assert q[0] == 0 and np.all(np.abs(q - want) <= abs(num) * f.tiny)
    for b in (f.tiny, 2 * f.tiny, 1.5 * f.tiny, edge / 2, 1.5 * edge / 4):
        a = np.array([0.75, -1.0, 0.7, 1.9], dt)
        assert np.array_equal(quotients(kind, a, np.full(4, b, dt)), a / b)
    # significands of all ones: exact quotients next to a tie, so at most one unit of the last place
    for b in (np.nextafter(edge, dt(0)), np.nextafter(dt(1), dt(0)), np.nextafter(dt(2) ** dt(30), dt(0))):
        a = np.array([0.75, -1.0, 0.7], dt)
        assert np.all(np.abs(quotients(kind, a, np.full(3, b, dt)) - a / b) <= np.spacing(np.abs(a / b)))
    for b in (0.0, -0.0, f.tiny / 8, f.smallest_subnormal, np.nan):
        assert not np.any(np.isfinite(quotients(kind, np.array([0.75, -1.0, 2.0], dt), np.full(3, b, dt))))


@pytest.mark.parametrize("placement", [0, 1, 2])
def test_infinite_admittance_in_a_dc_batch(placement):
    """An outage that leaves an infinite diagonal entry pins that bus at angle zero: a finite solution."""
    from lightsim2grid_b200 import Plan, synthetic

    g, V = synthetic.make_grid(33, 52, 5, seed=33)
    Y = g.get_dcYbus()
    S = V * np.conj(g.get_Ybus() @ V)
    bus = int(g.get_pq()[0])
    plan = Plan(Y, V, S, g.get_slack_ids(), g.get_slack_weights(), g.get_pv(), g.get_pq(), dc=True,
                lu_placement=placement)
    Vo, conv, it, err = plan.batch_n1([[(bus, bus, complex(-np.inf, 0.0))]] * 2, V, S, 10, 1e-8)
    assert conv.all() and np.all(err == 0) and np.all(np.isfinite(Vo))
    keep = np.array([b for b in range(g.n_bus) if b != bus and b not in set(g.get_slack_ids())])
    B = Y.real.toarray()
    th = np.linalg.solve(B[np.ix_(keep, keep)], S.real[keep])
    got = np.angle(Vo[0] / Vo[0][g.get_slack_ids()[0]])
    assert abs(got[bus]) <= 1e-12 and np.abs(np.angle(np.exp(1j * (got[keep] - th)))).max() <= 1e-9
