"""mult! and mult_adjoint! over array ranks and band widths: the unrolled kernels (2 to 4
dimensions, narrow bands), their per-entry general form (wide bands) and the general
kernels (other ranks), against dense products in Float64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _banded(sg, rng, m, n, width, dtype):
    """A valid refinement matrix [m, n] (m >= n) whose rows have up to `width` columns."""
    A = np.zeros((m, n), dtype=dtype)
    for i in range(m):
        c0 = int(round(i * (n - 1) / max(m - 1, 1)))
        lo, hi = max(0, c0 - (width - 1) // 2), min(n, c0 + width // 2 + 1)
        A[i, lo:hi] = rng.uniform(0.1, 1.0, hi - lo)
    return sg.RefinementMatrix.from_dense(A)


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("sizes,dims,widths", [
    (((9, 17), (4, 4)), (0,), (2,)),                                   # rank 2, one dimension
    (((1, 1), (3, 3)), (0,), (1,)),                                    # one control point
    (((9, 17), (8, 15), (3, 3)), (0, 1), (3, 5)),                      # rank 3
    (((9, 9), (8, 15), (3, 3)), (1,), (9,)),                           # a wide band
    (((6, 11), (7, 13), (5, 9), (2, 2)), (0, 1, 2), (3, 3, 3)),        # rank 4
    (((6, 11), (7, 7), (5, 9), (2, 2)), (2, 0), (7, 2)),               # wide in a slow dimension
    (((30, 58), (30, 57), (14, 26), (1, 1)), (0, 1, 2), (2, 3, 4)),    # several blocks
    (((4, 7), (3, 3), (3, 5), (3, 5), (2, 2)), (0, 2, 3), (2, 3, 2)),  # rank 5: the general kernel
])
def test_mult_matches_dense(sg, dtype_name, sizes, dims, widths):
    import torch
    dt, npt = (torch.float64, np.float64) if dtype_name == "f64" else (torch.float32, np.float32)
    u = 2.0 ** -53 if dtype_name == "f64" else 2.0 ** -24
    rng = np.random.default_rng(len(sizes) * 100 + len(dims))
    nB, nY = [s[0] for s in sizes], [s[1] for s in sizes]
    mats = [_banded(sg, rng, nY[d], nB[d], w, npt) for d, w in zip(dims, widths)]
    B = rng.standard_normal(nB).astype(npt)
    Yb = rng.standard_normal(nY).astype(npt)
    Y = sg.arrays.empty(nY, dt)
    sg.mult_(Y, mats, sg.arrays.from_any(torch.as_tensor(B), dt), dims)
    Bb = sg.arrays.empty(nB, dt)
    sg.mult_adjoint_(Bb, mats, sg.arrays.from_any(torch.as_tensor(Yb), dt), dims)
    for got, x, adj in ((Y, B, False), (Bb, Yb, True)):
        ref, mag, terms = x.astype(np.float64), np.abs(x.astype(np.float64)), 1
        for A, d in zip(mats, dims):
            D = A.collect().astype(np.float64)
            D = D.T if adj else D
            ref = np.moveaxis(np.tensordot(D, ref, axes=(1, d)), 0, d)
            mag = np.moveaxis(np.tensordot(np.abs(D), mag, axes=(1, d)), 0, d)
            terms *= int((D != 0).sum(1).max())
        # `terms` products of len(dims) + 1 factors, summed one after the other
        bound = 1.01 * (terms + len(dims)) * u * mag
        assert np.all(np.abs(got.cpu().numpy().astype(np.float64) - ref) <= bound)
