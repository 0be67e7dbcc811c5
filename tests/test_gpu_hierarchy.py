"""The hierarchy build's frontier loops (kPairLoop, kDepthLoop in hierarchy.cu) where they take the most rounds:
a line of cells has about as many as cells, on every level, each behind a barrier of the whole grid.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from brae_b200 import cases  # noqa: E402


@pytest.mark.parametrize("n", [1023, 30011])
def test_line_of_cells(oracle, n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import brae_b200.native as b2g
    c = cases.box_case(n, 1, 1)
    mesh = b2g.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
    H = oracle.agglomerate(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True).hierarchy
    assert mesh.n_levels == H.n_levels
    for s in range(H.n_levels):
        st = mesh.step(s)
        assert np.array_equal(st["restrict"], H.restrict[s]), s
        assert np.array_equal(st["lower"], H.lower[s + 1]) and np.array_equal(st["upper"], H.upper[s + 1]), s
