"""The LU programs' FP64 quotient (a reciprocal instruction, Newton steps and a remainder correction
instead of the division operator): a DC power flow of a two-bus grid is one such quotient, theta = P / B,
over operands of very different sizes."""
import numpy as np
import pytest
from scipy import sparse

pytestmark = pytest.mark.gpu


def test_dc_angle_is_the_rounded_quotient():
    from lightsim2grid_b200 import Plan

    rng = np.random.default_rng(3)
    for _ in range(40):
        b = rng.uniform(1.0, 2.0) * 2.0 ** rng.integers(-40, 40)
        p = b * rng.uniform(1e-9, 0.5)
        Y = sparse.csc_matrix(np.array([[b, -b], [-b, b]], dtype=np.complex128))
        V0 = np.array([1.0 + 0j, 1.0 + 0j])
        plan = Plan(Y, V0, np.array([0, p + 0j]), np.array([0]), np.array([1.0, 0.0]), np.array([1]),
                    np.zeros(0, np.int64), dc=True)
        V, conv, _, _ = plan.solve(V0, np.array([-p + 0j, p + 0j]), 10, 1e-8)
        assert conv
        # angle of exp(j theta): sincos and arctan are a few ulp each
        assert abs(np.angle(V[1]) - p / b) <= 4e-16 * max(abs(p / b), 1e-9) + 2e-16 * abs(p / b)
