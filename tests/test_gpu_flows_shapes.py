"""Branch flows on both sides of every line of the launch rule: the branch count and row counts from which few
rows take wide CTAs (2 and 4 per SM of 148), and the row size from which all do."""
import pytest

from test_gpu_flows_edges import test_edges as _edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, rows", [(420, 200), (430, 200), (600, 296), (600, 297), (1600, 592), (1600, 593),
                                     (2124, 600), (2125, 600)])
def test_shapes(n, rows):
    _edges(n, rows)
