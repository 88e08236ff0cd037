"""The axis-0 adjoint tiles, single values and 16-byte groups: spans that start and end at every
offset within a group, supports longer than a staged segment, columns and control points that
leave a tile partly filled.  Both sum a control point's samples in increasing order with one
FMA each, so the passes must have the bits of the fused launch."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deg0", [0, 1, 2, 3])
@pytest.mark.parametrize("n0,ns0", [
    (37, 400),      # groups; spans of 10 to 12 samples
    (37, 401),      # single values
    (150, 452),     # spans of 3: groups that belong to several spans
    (9, 2000),      # spans longer than a segment
    (64, 64),       # a span per sample
])
def test_axis0_tiles_have_the_fused_bits(sg, deg0, n0, ns0):
    import torch
    # many columns so that the tiles run: 131 axis-1 control points x 3, a group partly filled
    dims = (sg.SplineDimension(n0, deg0, ns0, float_type=torch.float32),
            sg.SplineDimension(131, 2, 300, float_type=torch.float32))
    g = sg.SplineGrid(dims, 3)
    plan = g.plan(torch.float32)
    cot = sg.arrays.empty((ns0, 300, 3), torch.float32)
    gen = torch.Generator(device="cuda").manual_seed(n0)
    cot.copy_(torch.randn((ns0, 300, 3), generator=gen, device="cuda"))
    cot[5, 7, 1] = float("inf")   # stays in its own supports
    got = []
    for strategy in ("fused", "separable"):
        plan.set_strategy(strategy)
        gr = sg.arrays.empty((n0, 131, 3), torch.float32)
        gr.fill_(float("nan"))
        sg.evaluate_adjoint_(g, control_points=gr, eval=cot)
        plan.check()
        got.append(gr)
    assert torch.isfinite(got[0]).sum() > 0.9 * got[0].numel()
    assert torch.equal(torch.nan_to_num(got[0], nan=1.5), torch.nan_to_num(got[1], nan=1.5))


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("n0,ns0,n1,nout", [
    (5, 1000, 4, 1),     # four columns, supports of 600 samples and more: a tile
    (5, 1001, 5, 2),
    (300, 600, 4, 1),    # supports of six: one thread per output
    (900, 1500, 4, 1),
    (40, 900, 4, 5),     # 20 columns of one tile
])
def test_few_columns_have_the_fused_bits(sg, n0, ns0, n1, nout, dtype_name):
    import torch
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    g = sg.SplineGrid((sg.SplineDimension(n0, 2, ns0, float_type=dt),
                       sg.SplineDimension(n1, 1, 30, float_type=dt)), nout)
    plan = g.plan(dt)
    gen = torch.Generator(device="cuda").manual_seed(n0 + n1)
    cot = sg.arrays.empty((ns0, 30, nout), dt)
    cot.copy_(torch.randn((ns0, 30, nout), generator=gen, device="cuda", dtype=dt))
    got = []
    for strategy in ("fused", "separable"):
        plan.set_strategy(strategy)
        gr = sg.arrays.empty((n0, n1, nout), dt)
        gr.fill_(float("nan"))
        sg.evaluate_adjoint_(g, control_points=gr, eval=cot)
        plan.check()
        got.append(gr)
    assert torch.isfinite(got[0]).all()
    assert torch.equal(got[0], got[1])
