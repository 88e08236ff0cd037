"""The per-grid separable passes over the sizes where their kernels change or end: one
thread per output, 32-column units, rings of 16-byte lanes, axis-0 tiles; degrees 0 to 6;
rows off the 16-byte lines; unsorted samples; more control points than samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n_control, degree, n_samples, nout, sorted)
SHAPES = [
    ((7, 6), (4, 5), (41, 33), 2, True),            # one thread per output, degrees 4 and 5
    ((9, 8), (6, 3), (33, 29), 1, True),            # degree 6: the runtime-degree kernels
    ((5, 4, 6), (0, 3, 2), (9, 1, 14), 1, True),    # a single sample
    ((10, 8), (3, 2), (64, 50), 3, False),          # unsorted samples
    ((40, 24), (3, 3), (1028, 1024), 1, True),      # just above the thread limit: ring
    ((40, 24), (3, 4), (1029, 1023), 1, True),      # 32-column units, rows off the lines
    ((33, 400), (2, 2), (4104, 260), 1, True),      # more control points than samples
    ((300, 9), (1, 3), (2052, 523), 1, True),       # few, long spans along axis 1
    ((20, 30), (5, 2), (1032, 1030), 1, False),     # unsorted, large
    ((12, 11, 19), (2, 3, 4), (64, 68, 250), 1, True),   # three passes above the limit
    ((64, 16), (2, 2), (8192, 131), 1, True),       # axis-0 supports longer than a tile segment
    ((9,), (2,), (600,), 3, True),                  # curves: just short of and beyond the split sum,
    ((9,), (3,), (700,), 1, False),
    ((200,), (3,), (20011,), 2, True),              # one CTA per control point,
    ((8,), (5,), (30001,), 3, True),                # and clusters
    ((6,), (0,), (2 ** 17 + 3,), 5, False),
]


@pytest.mark.parametrize("dtype_name", ["f32", "f64"])
@pytest.mark.parametrize("si", range(len(SHAPES)))
def test_separable_passes_match_oracle(sg, oracle, dtype_name, si):
    import torch
    from test_gpu_parity import oracle_spec
    n, deg, ns, nout, is_sorted = SHAPES[si]
    dt = torch.float64 if dtype_name == "f64" else torch.float32
    u = 2.0 ** -53 if dtype_name == "f64" else 2.0 ** -24
    rng = np.random.default_rng(40 + si)
    dims = tuple(sg.SplineDimension(a, b, c, float_type=dt,
                                    sample_points=None if is_sorted else rng.random(c))
                 for a, b, c in zip(n, deg, ns))
    g = sg.SplineGrid(dims, nout)
    plan = g.plan(dt)
    plan.set_strategy("separable")
    cp = rng.standard_normal(n + (nout,))
    cot = rng.standard_normal(ns + (nout,))
    cp_t, cot_t = (sg.arrays.from_any(torch.as_tensor(x), dt) for x in (cp, cot))
    ev = sg.arrays.empty(ns + (nout,), dt)
    ev.fill_(float("nan"))
    gr = sg.arrays.empty(n + (nout,), dt)
    gr.fill_(float("nan"))
    sg.evaluate_(g, control_points=cp_t, eval=ev)
    sg.evaluate_adjoint_(g, control_points=gr, eval=cot_t)
    plan.check()
    spec = oracle_spec(oracle, g)
    cp64 = np.asfortranarray(cp_t.cpu().numpy().astype(np.float64))
    cot64 = np.asfortranarray(cot_t.cpu().numpy().astype(np.float64))
    # rounding of a sum of k products is at most k u times the sum of the magnitudes; each
    # axis adds its terms, and each rounded basis table one u (a few for its own recursion)
    support = 0
    for dim, m, d in zip(dims, n, deg):  # samples per knot span, then per control point
        spans = np.bincount(dim.sample_indices.cpu().numpy() - d - 1, minlength=m - d)
        support += int(np.convolve(spans, np.ones(d + 1, dtype=np.int64)).max())
    k_f, k_a = sum(d + 1 for d in deg) + 8 * len(n), support + 8 * len(n)
    ref, mag = oracle.evaluate(spec, cp64), oracle.evaluate(spec, np.abs(cp64))
    assert np.all(np.abs(ev.cpu().numpy() - ref) <= 1.01 * k_f * u * mag)
    ref, mag = oracle.evaluate_adjoint(spec, cot64), oracle.evaluate_adjoint(spec, np.abs(cot64))
    assert np.all(np.abs(gr.cpu().numpy() - ref) <= 1.01 * k_a * u * mag)
    # the same bits again
    again = sg.arrays.empty(n + (nout,), dt)
    sg.evaluate_adjoint_(g, control_points=again, eval=cot_t)
    assert torch.equal(gr, again)


def test_large_adjoint_on_two_streams(sg):
    """Large 2D adjoints of one plan in flight on two streams, and captured: the bits of a
    call alone."""
    import torch
    dims = tuple(sg.SplineDimension(a, 3, s) for a, s in ((60, 2048), (50, 1100)))
    g = sg.SplineGrid(dims, 1)
    plan = g.plan(torch.float32)
    assert plan.paths() == ("fused", "separable")
    gen = torch.Generator(device="cuda").manual_seed(1)
    cots = [torch.randn((1, 1100, 2048), device="cuda", generator=gen).permute(2, 1, 0) for _ in range(6)]
    outs = [sg.arrays.empty((60, 50, 1), torch.float32) for _ in cots]
    refs = [sg.arrays.empty((60, 50, 1), torch.float32) for _ in cots]
    for c, r in zip(cots, refs):
        sg.evaluate_adjoint_(g, eval=c, control_points=r)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for k, (c, o) in enumerate(zip(cots, outs)):
        with torch.cuda.stream(streams[k % 2]):
            sg.evaluate_adjoint_(g, eval=c, control_points=o)
    torch.cuda.synchronize()
    assert all(torch.equal(o, r) for o, r in zip(outs, refs))
    outs[0].zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sg.evaluate_adjoint_(g, eval=cots[0], control_points=outs[0])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(outs[0], refs[0])
    plan.check()


def test_batch_curves_equal_per_grid(sg):
    """Curves with long and short supports in one batch with a surface: the bits of the
    per-grid calls."""
    import torch
    sizes = [(((12,), (3,)), (5000,)), (((40,), (2,)), (100,)), (((9, 8), (2, 2)), (30, 40)), (((7,), (1,)), (3000,))]
    grids, cots, grads = [], [], []
    gen = torch.Generator(device="cuda").manual_seed(4)
    for (n, d), s in sizes:
        dims = tuple(sg.SplineDimension(a, b, c) for a, b, c in zip(n, d, s))
        g = sg.SplineGrid(dims, 2)
        grids.append(g)
        cots.append(torch.randn((2,) + s[::-1], device="cuda", generator=gen).permute(*reversed(range(len(s) + 1))))
        grads.append(sg.arrays.empty(n + (2,), torch.float32))
    batch = sg.GridBatch(grids)
    batch.set_arrays(None, None, cots, grads)
    batch.run(forward=False, adjoint=True)
    batch.check()
    for g, c, got in zip(grids, cots, grads):
        ref = sg.arrays.empty(tuple(got.shape), torch.float32)
        sg.evaluate_adjoint_(g, eval=c, control_points=ref)
        assert torch.equal(got, ref)
