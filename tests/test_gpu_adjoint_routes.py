"""The kernels of a separable adjoint pass on both sides of the lines between them: short and long
rows, few and many samples a control point, aligned and not, sorted and not.  All sum a control
point's samples in the same order, so the result has the bits of the batch's pass queue, which
chooses among other kernels by other rules; and it is the oracle's to a derived bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n_control, degree, n_samples, nout): the axis-1 pass has rows of n_samples[0] values, the axis-0
# pass n_control[1] * nout columns
SHAPES = [
    ((5, 40), (2, 3), (17, 300), 3),            # rows below 24 values
    ((4, 20), (1, 3), (8, 4000), 1),            # the same, few outputs with long sums
    ((4, 20), (3, 2), (9, 4000), 1),
    ((6, 70000), (3, 1), (16, 80000), 1),       # hardly a sample a control point; 70000 columns
    ((9, 20000), (1, 1), (16, 18000), 1),
    ((30, 50), (3, 3), (64, 100), 2),           # short sums, small
    ((100, 100), (3, 2), (3000, 150), 1),       # short sums, warp tasks
    ((90, 100), (1, 2), (3001, 150), 1),
    ((90, 100), (2, 4), (3000, 150), 1),        # degree 4: rings, columns
    ((700, 20), (2, 3), (9000, 100), 1),        # long sums; Float64 columns
    ((3, 4), (0, 2), (270000, 20), 1),          # many columns of few samples
    ((500, 30), (2, 1), (16389, 150), 1),       # unaligned rows, sums below 16
    ((20, 50), (2, 1), (60, 500), 1),           # axis 0: few outputs
    ((300, 2000), (3, 2), (600, 2100), 2),      # axis 0: many outputs, S = 8
    ((3, 11000), (2, 1), (40, 12000), 3),       # axis 0: 33000 columns of 40 samples
    ((20000, 4), (3, 1), (120000, 12), 2),      # axis 0: 8 columns
    ((2000, 50), (3, 2), (4000, 60), 2),        # axis 0: Float64 warp tasks
    ((3, 15000), (1, 1), (14, 16000), 2),
    ((60, 600), (2, 5), (2000, 640), 1),        # 600 chunks and more
    ((200, 300), (4, 2), (2100, 900), 7),       # degree 4 on axis 0
    ((1300, 900), (1, 1), (1200, 950), 1),      # axis 0: hardly a sample, many outputs
    ((60, 180), (2, 1), (9000, 1000), 1),       # unsorted: warp tasks both ways
]


@pytest.mark.parametrize("unsorted", [False, True])
@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("si", range(len(SHAPES)))
def test_pass_kernels_agree(sg, oracle, dtype_name, unsorted, si):
    import torch
    from test_gpu_parity import oracle_spec
    n, deg, ns, nout = SHAPES[si]
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    rng = np.random.default_rng(si)
    dims = tuple(sg.SplineDimension(a, d, s, float_type=dt, sample_points=rng.random(s) if unsorted else None)
                 for a, d, s in zip(n, deg, ns))
    g = sg.SplineGrid(dims, nout)
    plan = g.plan(dt)
    plan.set_strategy("separable")
    cot = sg.arrays.from_any(torch.as_tensor(rng.standard_normal(ns + (nout,))), dt)
    got = sg.arrays.empty(n + (nout,), dt)
    got.fill_(float("nan"))
    sg.evaluate_adjoint_(g, eval=cot, control_points=got)
    assert bool(torch.isfinite(got).all())
    if max(deg) <= 3:
        batch = sg.GridBatch([g])
        batch.set_strategy("separable")
        grad = sg.arrays.zeros(n + (nout,), dt)
        batch.set_arrays([sg.arrays.zeros(n + (nout,), dt)], [sg.arrays.empty(ns + (nout,), dt)], [cot], [grad])
        batch.run(forward=False, adjoint=True)
        batch.check()
        assert torch.equal(got, grad)
    # |result - exact| <= u * (multiply-adds of the longest chains + the basis values' own error) *
    # sum of the terms' magnitudes; a basis value's error is a few units a degree, magnified by the
    # number of spans, against weights that are 1 / (d + 1) on average
    spec = oracle_spec(oracle, g)
    cot64 = np.asfortranarray(cot.cpu().numpy().astype(np.float64))
    ref = oracle.evaluate_adjoint(spec, cot64)
    mag = oracle.evaluate_adjoint(spec, np.abs(cot64))
    u = 2.0 ** (-53 if dtype_name == "f64" else -24)
    steps = sum(ns) + sum(8 * (d + 1) ** 2 * (a + 1) for a, d in zip(n, deg))
    floor = u * steps * float(np.abs(cot64).max())  # control points whose terms all but vanish
    assert (np.abs(got.cpu().numpy() - ref) <= u * steps * mag + floor).all()
