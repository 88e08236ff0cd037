"""Forward passes over an axis k >= 1 cut into tasks of 4 to 32 samples, and the rational last
pass: runs of samples that end at, before and after a task's and a warp's 32 rows, aligned and
odd row lengths, one to three channels and one too many, against the oracle in Float64.

Tolerance, per value: the basis values of an axis are non-negative and sum to one; each takes at
most 4 (d + 1) roundings in its own recursion and d + 1 in the sum it enters, so Nin axes err by
at most 5 Nin (d + 1) u max |P|, u = 2^-24 or 2^-53.  A NURBS value is the quotient of two such
sums, whose terms carry weights within a factor of four: eight times that.  One d more covers the
rounding of products and quotient."""
import numpy as np
import pytest

from test_gpu_parity import make_grid, oracle_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,u", [("f32", 2.0 ** -24), ("f64", 2.0 ** -53)])
@pytest.mark.parametrize("n_cp,deg,ns,nout,nurbs", [
    ((9, 8), (2, 3), (36, 4), 1, True),          # one run of a task, M = 36: one partly filled warp
    ((9, 8), (2, 1), (131, 33), 3, True),        # a sample past the 32 rows, odd rows
    ((30, 20), (3, 0), (520, 129), 2, True),     # degree 0 on the last axis
    ((30, 6), (3, 3), (1024, 700), 1, True),     # runs longer than a task
    ((9, 40), (1, 2), (64, 41), 3, True),        # a new span at every sample
    ((6, 7, 5), (2, 2, 2), (24, 30, 33), 4, True),   # more channels than a task holds
    ((6, 7, 5), (2, 3, 2), (128, 70, 65), 1, False),
    ((6, 7, 40), (2, 1, 3), (67, 71, 130), 2, False),
    ((6, 7, 9), (1, 5, 4), (100, 90, 70), 1, False),
])
def test_forward_tasks(sg, oracle, n_cp, deg, ns, nout, nurbs, dtype, u):
    torch = pytest.importorskip("torch")
    g = make_grid(sg, n_cp, deg, ns, dtype, nout, seed=3)
    w = None
    if nurbs:
        w = np.random.default_rng(7).uniform(0.5, 2.0, n_cp)
        g.weights = sg.arrays.from_any(torch.as_tensor(w), g.dtype)
        w = g.weights.cpu().numpy().astype(np.float64)
    sg.evaluate_(g)
    cp = sg.obtain(g.control_points).cpu().numpy().astype(np.float64)
    ref = oracle.evaluate(oracle_spec(oracle, g), cp, weights=w)
    err = np.abs(g.eval.cpu().numpy().astype(np.float64) - ref).max()
    assert err <= 5 * len(n_cp) * (max(deg) + 2) * u * (8 if nurbs else 1) * np.abs(cp).max()
