"""A large 2D grid's adjoint runs as two passes through an intermediate of its plan: calls on
several streams, tuning beside them and captures keep each result apart."""
import pytest

pytestmark = pytest.mark.gpu

N, NS, NOUT = (96, 80), (2048, 1024), 1


def _large(sg):
    """A grid whose adjoint goes through the plan's intermediate, its cotangent and gradient."""
    import torch
    g = sg.SplineGrid(tuple(sg.SplineDimension(n, 3, s) for n, s in zip(N, NS)), NOUT)
    gen = torch.Generator().manual_seed(11)
    cot = sg.arrays.from_any(torch.randn(NS + (NOUT,), generator=gen), torch.float32)
    want = sg.arrays.empty(N + (NOUT,), torch.float32)
    sg.evaluate_adjoint_(g, eval=cot, control_points=want)
    torch.cuda.synchronize()
    assert g.plan(torch.float32).paths() == ("fused", "separable")
    return g, cot, want


def test_tuning_waits_for_another_streams_adjoints(sg):
    """sg_grid_plan_tune writes the intermediate that adjoints still queued on another stream read."""
    import torch
    g, cot, want = _large(sg)
    queued = [sg.arrays.zeros(N + (NOUT,), torch.float32) for _ in range(40)]
    other = sg.arrays.from_any(-cot, torch.float32)
    scratch = sg.arrays.empty(N + (NOUT,), torch.float32)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(2_000_000)  # the calls below are queued before any of them runs
        for q in queued:
            sg.evaluate_adjoint_(g, eval=cot, control_points=q)
    with torch.cuda.stream(b):
        sg.tune_adjoint_(g, eval=other, control_points=scratch)
    torch.cuda.synchronize()
    for q in queued:
        assert torch.equal(q, want)
    # and adjoints that follow the tuning, on the first stream
    with torch.cuda.stream(a):
        queued[0].zero_()
        sg.evaluate_adjoint_(g, eval=cot, control_points=queued[0])
    torch.cuda.synchronize()
    assert torch.equal(queued[0], want)
    g.plan(torch.float32).untune()
