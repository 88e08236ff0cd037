"""mult! and mult_adjoint! with a band width of its own for each dimension: the choice between unrolled
sums and loops depends on how many of the unrolled terms are missing.  Against dense products in
Float64; ranks 2 to 5."""
import numpy as np
import pytest

from test_gpu_mult_bands import _banded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("sizes,dims,widths", [
    (((11, 21), (9, 17), (3, 3)), (0, 1), (1, 3)),
    (((11, 21), (9, 17), (3, 3)), (0, 1), (2, 5)),
    (((11, 40), (3, 3)), (0,), (4,)),
    (((10, 19), (11, 20), (9, 10), (2, 2)), (0, 1, 2), (1, 3, 2)),
    (((10, 19), (11, 20), (9, 10), (2, 2)), (0, 1, 2), (4, 3, 5)),
    (((10, 19), (11, 20), (9, 10), (2, 2)), (0, 1, 2), (2, 6, 1)),
    (((10, 19), (11, 20), (9, 10), (2, 2)), (0, 1, 2), (3, 3, 3)),
    (((10, 10), (11, 11), (9, 18), (2, 2)), (2,), (3,)),
    (((6, 9), (5, 8), (7, 7), (6, 11), (2, 2)), (0, 1, 3), (2, 3, 4)),
])
def test_mixed_widths(sg, dtype_name, sizes, dims, widths):
    import torch
    dt, npt = (torch.float64, np.float64) if dtype_name == "f64" else (torch.float32, np.float32)
    u = 2.0 ** -53 if dtype_name == "f64" else 2.0 ** -24
    rng = np.random.default_rng(sum(widths))
    nB, nY = [s[0] for s in sizes], [s[1] for s in sizes]
    mats = [_banded(sg, rng, nY[d], nB[d], w, npt) for d, w in zip(dims, widths)]
    B, Yb = rng.standard_normal(nB).astype(npt), rng.standard_normal(nY).astype(npt)
    Y, Bb = sg.arrays.empty(nY, dt), sg.arrays.empty(nB, dt)
    Y.fill_(float("nan"))
    Bb.fill_(float("nan"))
    sg.mult_(Y, mats, sg.arrays.from_any(torch.as_tensor(B), dt), dims)
    sg.mult_adjoint_(Bb, mats, sg.arrays.from_any(torch.as_tensor(Yb), dt), dims)
    for got, x, adj in ((Y, B, False), (Bb, Yb, True)):
        ref, mag, terms = x.astype(np.float64), np.abs(x.astype(np.float64)), 1
        for A, d in zip(mats, dims):
            D = A.collect().astype(np.float64)
            D = D.T if adj else D
            ref = np.moveaxis(np.tensordot(D, ref, axes=(1, d)), 0, d)
            mag = np.moveaxis(np.tensordot(np.abs(D), mag, axes=(1, d)), 0, d)
            terms *= int((D != 0).sum(1).max())
        # terms products of len(dims) + 1 factors, summed one after the other, and as much
        # again for the Float64 reference's own sums
        bound = 1.01 * (terms + len(dims)) * (u + 2.0 ** -53) * mag
        assert np.all(np.abs(got.cpu().numpy().astype(np.float64) - ref) <= bound)
