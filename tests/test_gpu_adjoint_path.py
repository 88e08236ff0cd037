"""The path AUTO takes for the adjoint of large 2D grids: two passes where fused tiles re-read much
or sum in long chains, the tiles where the passes' intermediate is a large part of the cotangent.
Each shape is well on its side (the other path measured 1.3 to 3 times as long); both paths give
the same bits."""
import pytest

pytestmark = pytest.mark.gpu

# n_control, degree, n_samples, nout, dtype, path
SHAPES = [
    ((256, 256), (3, 3), (4096, 4096), 3, "f64", "separable"),   # long rows, 16 samples a point
    ((128, 128), (3, 3), (2048, 2048), 1, "f32", "separable"),
    ((327, 341), (3, 3), (32768, 1025), 1, "f32", "separable"),  # long sums along axis 0
    ((2255, 6), (0, 3), (16384, 646), 1, "f32", "separable"),    # few tiles
    ((8192, 256), (2, 2), (32768, 1024), 1, "f32", "fused"),     # a quarter of the values in between
    ((512, 1536), (2, 2), (2048, 6145), 1, "f32", "fused"),
    ((20, 341), (3, 3), (2048, 1025), 1, "f32", "fused"),        # three samples a point on axis 1
    ((81, 28), (3, 3), (8192, 86), 3, "f32", "fused"),
    ((64, 64), (2, 2), (1024, 2000), 1, "f32", "fused"),         # rows shorter than two tiles
    ((64, 64), (3, 3), (2048, 1000), 1, "f32", "fused"),         # fewer than 2^21 values
]


@pytest.mark.parametrize("si", range(len(SHAPES)))
def test_path_and_bits(sg, si):
    import torch
    n, deg, ns, nout, dtype_name, path = SHAPES[si]
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    g = sg.SplineGrid(tuple(sg.SplineDimension(a, d, s, float_type=dt) for a, d, s in zip(n, deg, ns)), nout)
    plan = g.plan(dt)
    assert plan.paths()[1] == path
    cot = torch.randn((nout,) + ns[::-1], device="cuda", dtype=dt).permute(2, 1, 0)
    out = []
    for strategy in ("auto", "separable", "fused"):
        plan.set_strategy(strategy)
        got = sg.arrays.empty(n + (nout,), dt)
        got.fill_(float("nan"))
        fused = sg.load_library().sg_test_fused_adjoint_launches()
        sg.evaluate_adjoint_(g, eval=cot, control_points=got)
        launched = sg.load_library().sg_test_fused_adjoint_launches() - fused
        assert launched == (path == "fused" if strategy == "auto" else strategy == "fused")
        out.append(got)
    plan.check()
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


def test_tuning_keeps_the_path(sg):
    """Tuning may change a plan's tiles; the path stays that of the untuned ones, also after a refresh."""
    import torch
    for n, ns, path in (((96, 80), (2048, 1024), "separable"), ((20, 341), (2048, 1025), "fused")):
        g = sg.SplineGrid(tuple(sg.SplineDimension(a, 3, s) for a, s in zip(n, ns)), 1)
        plan = g.plan(torch.float32)
        assert plan.paths()[1] == path
        sg.tune_adjoint_(g, eval=g.eval)
        assert plan.paths()[1] == path
        g.refresh_plans()
        assert plan.paths()[1] == path
        plan.untune()
        assert plan.paths()[1] == path
