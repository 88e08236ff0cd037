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


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
def test_tuning_a_curve_runs_its_adjoint(sg, dtype_name):
    """A curve with long supports sums them with a kernel of its own, in another order than the
    passes over several columns do; the gradient that tuning leaves behind has its bits."""
    import torch
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    g = sg.SplineGrid((sg.SplineDimension(15, 3, 6001, float_type=dt),), 2)
    gen = torch.Generator().manual_seed(5)
    cot = sg.arrays.from_any(torch.randn((6001, 2), generator=gen, dtype=torch.float64), dt)
    want, left = sg.arrays.empty((15, 2), dt), sg.arrays.empty((15, 2), dt)
    sg.evaluate_adjoint_(g, eval=cot, control_points=want)
    assert sg.tune_adjoint_(g, eval=cot, control_points=left) == [0]
    assert torch.equal(left, want)


def test_tuning_a_large_grid_times_both_of_its_adjoints(sg):
    """A large 2D grid's adjoint is separable but for calls that cannot have the plan's intermediate
    (captured ones among them), which are fused: tuning runs both, and neither result changes."""
    import torch
    n, ns = (96, 80), (2048, 1024)
    g = sg.SplineGrid(tuple(sg.SplineDimension(a, 3, s) for a, s in zip(n, ns)), 1)
    plan, lib = g.plan(torch.float32), sg.load_library()
    assert plan.paths()[1] == "separable"
    gen = torch.Generator().manual_seed(6)
    cot = sg.arrays.from_any(torch.randn(ns + (1,), generator=gen), torch.float32)
    want, got, scratch = (sg.arrays.empty(n + (1,), torch.float32) for _ in range(3))
    sg.evaluate_adjoint_(g, eval=cot, control_points=want)
    plan.check()
    fused = lib.sg_test_fused_adjoint_launches()
    chosen = sg.tune_adjoint_(g, eval=cot, control_points=scratch)
    plan.check()
    assert lib.sg_test_fused_adjoint_launches() > fused
    assert chosen[0] == 0 and chosen[1] in (0, 8, 12, 16, 24, 32, 48, 64)  # the separable pass'
    sg.evaluate_adjoint_(g, eval=cot, control_points=got)
    assert torch.equal(got, want)
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    got.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s):
            sg.evaluate_adjoint_(g, eval=cot, control_points=got)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    plan.untune()
