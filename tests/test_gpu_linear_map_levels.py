"""A linear map made before its grid was refined further refuses its vectors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_map_from_before_a_refinement_is_refused(sg):
    import torch
    g = sg.SplineGrid(tuple(sg.SplineDimension(n, 2, s) for n, s in zip((8, 7), (40, 30))), 2)
    g = sg.add_default_local_refinement(g)
    sg.activate_local_refinement_(g.control_points, np.array([[3, 3], [4, 4]]))
    A = sg.LinearMap(g)
    x = torch.ones(A.shape[1], device="cuda")
    y = A @ x
    sg.activate_local_refinement_(g.control_points, np.array([[5, 5], [6, 6], [7, 5]]))
    with pytest.raises(AssertionError):
        A @ x
    with pytest.raises(AssertionError):
        A.T @ y
    B = sg.LinearMap(g)
    assert B.shape[1] == A.shape[1] + 3 * 2
    xb = torch.ones(B.shape[1], device="cuda")
    assert bool(torch.isfinite(B @ xb).all()) and bool(torch.isfinite(B.T @ y).all())
