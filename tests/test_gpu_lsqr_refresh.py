"""A solver made before its grid's samples moved (set_sample_indices_, evaluate_dimension_ and
refresh_plans) solves for the samples as they are: the solution of a solver made afterwards,
bit for bit; captured and not, with a plan of its own (a large grid) and without."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("n,ns,unsorted", [((24, 20), (2048, 1024), False), ((24, 20), (2048, 1024), True),
                                           ((9, 8), (60, 50), False), ((15,), (4000,), False)])
def test_a_solver_follows_its_grids_refresh(sg, n, ns, unsorted, graph):
    import torch
    dims = tuple(sg.SplineDimension(a, 3, s, float_type=torch.float64) for a, s in zip(n, ns))
    g = sg.SplineGrid(dims, 1)
    gen = torch.Generator().manual_seed(3)
    b = torch.randn(g.eval.numel(), generator=gen, dtype=torch.float64).cuda()
    A = sg.LinearMap(g)
    kw = dict(maxiter=6, atol=0.0, btol=0.0, conlim=0.0, graph=graph)
    solver = sg.LSQRSolver(A, **kw)
    before = solver.solve(b)
    dim = dims[-1]
    pts = dim.sample_points ** 1.5
    if unsorted:
        pts = pts.flip(0)
    dim.sample_points.copy_(pts)
    sg.set_sample_indices_(dim)
    sg.evaluate_dimension_(dim)
    g.refresh_plans()
    got = solver.solve(b)
    want = sg.LSQRSolver(sg.LinearMap(g), **kw).solve(b)
    assert not torch.equal(got, before)
    assert torch.equal(got, want)
