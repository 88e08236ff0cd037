"""Kernels whose set-up overlaps the end of the kernel before them: chains of passes that read what
the previous launch wrote, many in a row without a pause, give the bits of the same calls
with the stream drained after each; on the default stream, on another one and captured."""
import pytest

pytestmark = pytest.mark.gpu


def _chain(sg, grids, evals, grads, pause):
    """Evaluate, take the adjoint, and make the result the next round's control points."""
    import torch
    for r in range(6):
        for g, ev, gr in zip(grids, evals, grads):
            src = gr if r else sg.obtain(g.control_points)
            sg.evaluate_(g, control_points=src, eval=ev)
            if pause:
                torch.cuda.synchronize()
            sg.evaluate_adjoint_(g, control_points=gr, eval=ev)
            if pause:
                torch.cuda.synchronize()


@pytest.mark.parametrize("where", ["default", "stream", "graph"])
def test_back_to_back_launches_keep_their_order(sg, where):
    import torch
    shapes = [((10, 10, 5), (2, 3, 2), (50, 50, 25), 2, torch.float64),   # one thread per output
              ((12, 9, 8), (2, 2, 2), (65, 70, 131), 1, torch.float32),
              ((20, 30), (3, 2), (300, 401), 3, torch.float32),           # fused
              ((40,), (3,), (20001,), 2, torch.float32),                  # clusters
              ((64, 64), (2, 3), (1100, 1003), 2, torch.float64)]         # separable adjoint
    grids, evals, grads = [], [], []
    for n, deg, ns, nout, dt in shapes:
        g = sg.SplineGrid(tuple(sg.SplineDimension(a, b, c, float_type=dt) for a, b, c in zip(n, deg, ns)), nout)
        gen = torch.Generator().manual_seed(len(n) + ns[0])
        cp = sg.obtain(g.control_points)
        scale = 1.0
        for a, c in zip(n, ns):
            scale *= a / c   # keeps adjoint(evaluate(.)) near unit size
        cp.copy_(torch.randn(tuple(cp.shape), generator=gen, dtype=torch.float64).to(dt) * scale)
        grids.append(g)
        evals.append(sg.arrays.empty(ns + (nout,), dt))
        grads.append(sg.arrays.empty(n + (nout,), dt))
    _chain(sg, grids, evals, grads, pause=True)
    want = [x.clone() for x in evals + grads]
    for x in evals + grads:
        x.fill_(float("nan"))
    torch.cuda.synchronize()
    if where == "default":
        _chain(sg, grids, evals, grads, pause=False)
    else:
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            if where == "stream":
                _chain(sg, grids, evals, grads, pause=False)
            else:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=s):
                    _chain(sg, grids, evals, grads, pause=False)
                graph.replay()
    torch.cuda.synchronize()
    for g in grids:
        g.plan(evals[grids.index(g)].dtype).check()
    for got, ref in zip(evals + grads, want):
        assert torch.equal(got, ref)
