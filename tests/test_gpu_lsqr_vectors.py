"""The vector passes of the device LSQR: lengths that leave a remainder of the 16-byte groups, one
and two groups a thread, and a right-hand side whose address allows single values only,
against the oracle's LSQR after four iterations.

Tolerance of x, relative to its largest value: an iteration applies the operator and updates three
vectors, some 60 roundings of a value, and the quotients of the recurrence pass them on at most
tenfold here, so four iterations err by 4 * 60 * 10 u = 2400 u."""
import numpy as np
import pytest

from test_gpu_lsqr import _spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n,deg,ns,nout", [
    ((5,), (2,), (7,), 1),                  # fewer values than a group and a remainder
    ((7, 9), (2, 1), (31, 23), 1),          # odd lengths in both spaces
    ((9, 6), (3, 2), (26, 73), 3),
    ((31, 17), (2, 2), (901, 701), 1),      # two groups a thread, and a single value left over
])
def test_lsqr_vector_lengths(sg, oracle, n, deg, ns, nout, offset, dtype_name):
    import torch
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    u = 2.0 ** -53 if dtype_name == "f64" else 2.0 ** -24
    offset *= 1 if dtype_name == "f64" else 2   # 8 bytes past a 16-byte boundary
    g = sg.SplineGrid(tuple(sg.SplineDimension(a, b, c, float_type=dt) for a, b, c in zip(n, deg, ns)), nout)
    spec = _spec(oracle, g)
    cps, evs = n + (nout,), ns + (nout,)
    m = int(np.prod(evs))
    store = torch.as_tensor(np.random.default_rng(m).standard_normal(m + offset), device="cuda").to(dt)
    b = store[offset:]
    mv = lambda x: oracle.evaluate(spec, np.asfortranarray(x.reshape(cps, order="F"))).ravel(order="F")
    rmv = lambda y: oracle.evaluate_adjoint(spec, np.asfortranarray(y.reshape(evs, order="F"))).ravel(order="F")
    solver = sg.LSQRSolver(sg.LinearMap(g), atol=0.0, btol=0.0, conlim=0.0, maxiter=4)
    x = solver.solve(b)
    x_ref, _, itn, _ = oracle.lsqr(mv, rmv, b.cpu().numpy().astype(np.float64), int(np.prod(cps)), atol=0.0,
                                   btol=0.0, conlim=0.0, maxiter=4)
    assert solver.info()["iterations"] == itn == 4
    err = np.abs(x.cpu().numpy().astype(np.float64) - x_ref).max()
    assert err <= 2400 * u * np.abs(x_ref).max()
