"""The first pass of NURBS grids with few samples along axis 0: blocks of the axis' length, at the ends
of warps and blocks; one thread a channel and threads that walk several.  Against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("nout", [1, 3])
@pytest.mark.parametrize("ns0", [1, 2, 31, 32, 33, 127, 128, 129, 300])
def test_short_first_axis(sg, oracle, dtype_name, nout, ns0):
    import torch
    from test_gpu_parity import oracle_spec
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    for n, deg, ns in (((5, 9), (2, 3), (ns0, 40)), ((4, 300), (3, 1), (ns0, 311)), ((4, 5, 21), (1, 2, 2), (ns0, 7, 30))):
        g = sg.NURBSGrid(tuple(sg.SplineDimension(a, d, s, float_type=dt) for a, d, s in zip(n, deg, ns)), nout)
        rng = np.random.default_rng(ns0 + nout)
        cp = sg.arrays.from_any(torch.as_tensor(rng.standard_normal(n + (nout,))), dt)
        g.weights.copy_(sg.arrays.from_any(torch.as_tensor(rng.uniform(0.5, 2.0, n)), dt))
        g.eval.fill_(float("nan"))
        sg.evaluate_(g, control_points=cp)
        ref = oracle.evaluate(oracle_spec(oracle, g), np.asfortranarray(cp.cpu().numpy().astype(np.float64)),
                              weights=np.asfortranarray(g.weights.cpu().numpy().astype(np.float64)))
        # numerator and denominator: a chain of d + 1 multiply-adds an axis, basis values off by a few
        # units a degree, magnified by the number of spans; the quotient is at most max |P| and the
        # weights differ by a factor of four
        u = 2.0 ** (-53 if dtype_name == "f64" else -24)
        steps = 4 + sum(d + 2 + 8 * (d + 1) * (a + 1) for a, d in zip(n, deg))
        assert np.abs(g.eval.cpu().numpy() - ref).max() <= 2 * 4 * steps * u * np.abs(cp.cpu().numpy()).max()
