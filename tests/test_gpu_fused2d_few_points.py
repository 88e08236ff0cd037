"""The fused adjoint with one control point (and other very few) on axis 0 and several channels
in a tile, and with more control points on axis 0 than a tile stages: against the oracle, and
against the separable passes bit for bit; the same through a batch and through autograd."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n_control, degree, n_samples)
SHAPES = [
    ((1, 9), (0, 2), (50, 41)),
    ((1, 6), (0, 3), (500, 30)),    # one channel a tile in Float64
    ((1, 1), (0, 0), (7, 5)),
    ((2, 9), (0, 2), (50, 41)),
    ((2, 7), (1, 1), (33, 40)),
    ((3, 5), (2, 3), (40, 60)),
    ((513, 8), (1, 2), (100, 33)),  # one more than is staged
    ((700, 12), (2, 1), (160, 50)),
]


def _oracle_grid(oracle, g):
    from test_gpu_parity import oracle_spec
    return oracle_spec(oracle, g)


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("nout", [1, 2, 3, 17])
@pytest.mark.parametrize("si", range(len(SHAPES)))
def test_adjoint_against_the_oracle_on_every_route(sg, oracle, dtype_name, nout, si):
    import torch
    n, deg, ns = SHAPES[si]
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    g = sg.SplineGrid(tuple(sg.SplineDimension(a, d, s, float_type=dt) for a, d, s in zip(n, deg, ns)), nout)
    rng = np.random.default_rng(si * 100 + nout)
    cot = sg.arrays.from_any(torch.as_tensor(rng.standard_normal(ns + (nout,))), dt)
    plan = g.plan(dt)
    assert plan.paths() == ("fused", "fused")
    want = {}
    for strategy in ("separable", "fused"):
        plan.set_strategy(strategy)
        out = sg.arrays.empty(n + (nout,), dt)
        out.fill_(float("nan"))
        sg.evaluate_adjoint_(g, eval=cot, control_points=out)
        plan.check()
        want[strategy] = out
    plan.set_strategy("auto")
    assert torch.equal(want["fused"], want["separable"])

    cot64 = cot.cpu().numpy().astype(np.float64)
    ref = oracle.evaluate_adjoint(_oracle_grid(oracle, g), np.asfortranarray(cot64))
    # A value is two chains of at most ns multiply-adds; a basis value is off by a few units for
    # each degree, times the samples' and knots' own rounding, which a knot span's width
    # magnifies by the number of spans.  All weights are at most 1.
    u = 2.0 ** (-53 if dtype_name == "f64" else -24)
    steps = ns[0] + ns[1] + sum(8 * (d + 1) * (a + 1) for a, d in zip(n, deg))
    bound = steps * u * np.abs(cot64).sum(axis=(0, 1))
    assert (np.abs(want["fused"].cpu().numpy() - ref) <= bound).all()

    # a batch of this grid and one more
    other = sg.SplineGrid(tuple(sg.SplineDimension(a, 2, s, float_type=dt) for a, s in ((8, 40), (9, 60))), 2)
    grids, shapes = [g, other], [n + (nout,), (8, 9, 2)]
    cots = [cot, sg.arrays.from_any(torch.as_tensor(rng.standard_normal((40, 60, 2))), dt)]
    grads = [sg.arrays.zeros(s, dt) for s in shapes]
    batch = sg.GridBatch(grids)
    batch.set_arrays([sg.arrays.zeros(s, dt) for s in shapes], [sg.arrays.empty(tuple(c.shape), dt) for c in cots],
                     cots, grads)
    batch.run(forward=False, adjoint=True)
    batch.check()
    assert torch.equal(grads[0], want["fused"])

    # autograd: the gradient of <cot, evaluate(cp)>
    cp = sg.arrays.zeros(n + (nout,), dt).requires_grad_()
    from splinegrids import autograd
    (autograd.evaluate(g, cp) * cot).sum().backward()
    assert torch.equal(cp.grad, want["fused"])
