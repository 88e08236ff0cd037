"""sg_grid_plan_tune times the configurations that later calls can take, the untuned one among
them."""
import pytest

pytestmark = pytest.mark.gpu


def test_tuning_can_keep_the_untuned_chunks(sg):
    """A long axis with a wide halo behind many rows: the untuned pass takes more control points a
    chunk than any of the sizes that are tried, and is the faster one (660 us against 678)."""
    import torch
    n, deg, ns = (20, 20, 500), (2, 2, 5), (1000, 600, 500)
    g = sg.SplineGrid(tuple(sg.SplineDimension(a, d, s) for a, d, s in zip(n, deg, ns)), 1)
    cot = sg.arrays.zeros(ns + (1,), torch.float32)
    grad = sg.arrays.empty(n + (1,), torch.float32)
    assert any(sg.tune_adjoint_(g, eval=cot, control_points=grad)[2] == 0 for _ in range(3))
