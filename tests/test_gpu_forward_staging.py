"""Fused forward tiles whose control points are staged, and those on the other side of each condition:
the bits of the separable passes."""
import pytest

pytestmark = pytest.mark.gpu

# n_control, degree, n_samples, nout, axis-0 samples sorted
SHAPES = [
    ((200, 200), (3, 3), (6000, 300), 4, True),   # many columns, a block that just fits
    ((100, 1600), (3, 2), (5600, 1900), 1, True),
    ((64, 2300), (2, 0), (2228, 3800), 3, True),
    ((64, 2300), (2, 0), (2229, 3800), 3, True),  # rows off the 16-byte boundaries
    ((256, 256), (3, 3), (4096, 4096), 1, True),   # long tiles of some 20 columns
    ((2000, 600), (3, 2), (4096, 1000), 1, True),  # blocks too large
    ((200, 200), (3, 3), (6000, 300), 4, False),
    ((300, 3), (2, 2), (200000, 5), 1, True),     # few rows
]


@pytest.mark.parametrize("dtype_name", ["f32", "f64", "bf16"])
@pytest.mark.parametrize("si", range(len(SHAPES)))
def test_forward_bits(sg, dtype_name, si):
    import torch
    n, deg, ns, nout, is_sorted = SHAPES[si]
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    gen = torch.Generator().manual_seed(si)
    pts = None if is_sorted else torch.rand(ns[0], generator=gen, dtype=torch.float64)
    g = sg.SplineGrid((sg.SplineDimension(n[0], deg[0], ns[0], float_type=dt, sample_points=pts),
                       sg.SplineDimension(n[1], deg[1], ns[1], float_type=dt)), nout)
    cp = sg.arrays.from_any(torch.randn(n + (nout,), generator=gen, dtype=torch.float64),
                            torch.bfloat16 if dtype_name == "bf16" else dt)
    plan = g.plan(cp.dtype)
    assert plan.paths()[0] == "fused"
    out = []
    for strategy in ("separable", "fused"):
        plan.set_strategy(strategy)
        ev = sg.arrays.empty(ns + (nout,), dt)
        ev.fill_(float("nan"))
        sg.evaluate_(g, control_points=cp, eval=ev)
        out.append(ev)
    plan.set_strategy("auto")
    assert torch.equal(out[0], out[1])
