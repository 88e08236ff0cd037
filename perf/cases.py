"""Performance cases: the work a user of the package has it do, through its public entry
points, over the sizes, types and options it takes.

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges, ``prepare`` what a
program holds before the call (grids with their plans, control points, cotangents), ``run``
one pass, ``work`` the bytes and operations a pass cannot do without, and ``exact`` the same
outputs in Float64 with plain torch and numpy.

Kinds of case:

* ``grid``: one spline grid (curve, surface or volume; plain, with first derivatives, NURBS,
  Float32, Float64 or bfloat16-stored control points): evaluate!, evaluate_adjoint!, or both,
  as an optimisation loop calls them; ``autograd`` goes through the differentiable call;
* ``refined``: a locally refined volume as a linear map, applied and its adjoint applied (what
  one step of a fit on truncated hierarchical splines does);
* ``batch``: many uneven surfaces, each with several control-point sets, forward and adjoint in
  one call;
* ``fit``: a least-squares fit of a surface with a fixed budget of LSQR iterations.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "splinegrids.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import splinegrids as sg  # noqa: E402


# ------------------------------------------------------------------------------ cases
def _grid(name, n, d, s, nout, dtype="f32", orders="value", way="both", nurbs=False, autograd=False):
    c = {"name": name, "kind": "grid", "nin": len(n), "nout": nout, "dtype": dtype, "orders": orders,
         "way": way, "nurbs": nurbs, "autograd": autograd}
    for k in range(len(n)):
        c["n%d" % k], c["d%d" % k], c["s%d" % k] = int(n[k]), int(d[k]), int(s[k])
    return c


def _refined(name, n, d, s, nout, levels, dtype="f32"):
    c = _grid(name, n, d, s, nout, dtype)
    c.update(kind="refined", levels=levels)
    return c


def listed():
    return [
        # a long planar path sampled finely, value and gradient of a loss on its points
        _grid("curve", (200,), (3,), (100001,), 2),
        # the README's volume: the smallest call, where launches and host work count
        _grid("volume_readme", (10, 10, 5), (2, 3, 2), (50, 50, 25), 4, dtype="f64"),
        # a heightfield of the size an interactive fit evaluates on each step
        _grid("heightfield", (64, 64), (2, 2), (1024, 1024), 1),
        # the large surface with both first derivatives (lens design): forward and adjoint
        _grid("surface_orders", (256, 256), (3, 3), (4096, 4096), 3, orders="gradient"),
        # the same surface in Float64
        _grid("surface_f64", (256, 256), (3, 3), (4096, 4096), 3, dtype="f64"),
        # bfloat16-stored control points: rendering a stored surface
        _grid("surface_bf16", (256, 256), (3, 3), (4096, 4096), 3, dtype="bf16", way="forward"),
        # an image-sized surface with odd extents inside a torch training step
        _grid("surface_odd", (97, 131), (3, 2), (1999, 1501), 3, autograd=True),
        # degrees above three (the reference's fits use (3, 4))
        _grid("surface_quartic", (120, 100), (3, 4), (1040, 731), 3, dtype="f64"),
        # a NURBS volume, evaluated
        _grid("volume_nurbs", (48, 48, 32), (2, 2, 2), (320, 320, 192), 1, way="forward", nurbs=True),
        # three levels of local refinement on a volume, applied and its adjoint
        _refined("volume_refined", (16, 16, 8), (2, 2, 2), (512, 512, 256), 1, 3),
        # many uneven surfaces with 16 control-point sets each, forward and adjoint
        {"name": "batch_uneven", "kind": "batch", "grids": 32, "sets": 16, "first": 5, "smax": 1024},
        # a least-squares fit of a surface to a scattered-noise heightfield
        {"name": "fit_surface", "kind": "fit", "n0": 256, "n1": 256, "d0": 3, "d1": 3, "s0": 2048, "s1": 2048,
         "nout": 1, "dtype": "f32", "iterations": 12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["curve", "surface", "surface", "surface", "surface", "volume", "volume", "refined",
                       "batch", "fit"])
    if kind == "curve":
        d = rng.choice([1, 2, 3, 3, 4, 5])
        c = _grid("", (_log(rng, d + 8, 2000),), (d,), (_log(rng, 300, 1000000),), rng.choice([1, 2, 3]),
                  dtype=rng.choice(["f32", "f32", "f64"]), orders=rng.choice(["value", "gradient"]))
    elif kind == "surface":
        d = [rng.choice([1, 2, 3, 3]) for _ in range(2)]
        if rng.random() < 0.15:
            d[rng.randrange(2)] = rng.choice([4, 5])
        dtype = rng.choice(["f32", "f32", "f64", "bf16"])
        orders = rng.choice(["value", "value", "gradient"])
        n = [_log(rng, 8, 256) for _ in range(2)]
        most = 1500 if max(d) > 3 else 2800 if dtype == "f64" and orders == "gradient" else 4096
        s = [_log(rng, 64, most) for _ in range(2)]
        if rng.random() < 0.5:
            s = [max(64, x - x % 8) for x in s]
        auto = dtype != "bf16" and orders == "value" and rng.random() < 0.3
        way = "forward" if dtype == "bf16" else "both" if auto else rng.choice(["forward", "adjoint", "both", "both"])
        c = _grid("", n, d, s, rng.choice([1, 2, 3, 4]) if s[0] * s[1] < 2 ** 22 else rng.choice([1, 3]),
                  dtype=dtype, orders=orders, way=way, autograd=auto)
    elif kind in ("volume", "refined"):
        d = [rng.choice([1, 2, 2, 3]) for _ in range(3)]
        if kind == "refined":
            levels = rng.choice([1, 2, 3])
            n = [rng.randint(d[k] + 3, 16) for k in range(3)]
            s = [_log(rng, 48, 400) for _ in range(3)]
            c = _refined("", n, d, s, rng.choice([1, 3]) if s[0] * s[1] * s[2] < 2 ** 23 else 1, levels)
        else:
            n = [rng.randint(5, 64) for _ in range(3)]
            s = [_log(rng, 24, 320) for _ in range(3)]
            nurbs = rng.random() < 0.5
            c = _grid("", n, d, s, rng.choice([1, 3, 4]) if s[0] * s[1] * s[2] < 2 ** 22 else 1,
                      dtype=rng.choice(["f32", "f32", "f64"]), nurbs=nurbs,
                      way="forward" if nurbs else rng.choice(["forward", "adjoint", "both"]))
    elif kind == "batch":
        c = {"kind": "batch", "grids": _log(rng, 2, 32), "sets": rng.choice([1, 4, 16]),
             "first": rng.randrange(100, 1000000), "smax": rng.choice([256, 512, 800])}
    else:
        dtype = rng.choice(["f32", "f64"])
        most = 2048 if dtype == "f32" else 1200
        c = {"kind": "fit", "n0": _log(rng, 16, 256), "n1": _log(rng, 16, 256), "d0": rng.choice([2, 3]),
             "d1": rng.choice([2, 3]), "s0": _log(rng, 520, most), "s1": _log(rng, 520, most), "nout": 1,
             "dtype": dtype, "iterations": rng.choice([4, 8, 12])}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------ inputs
_DT = {"f32": torch.float32, "f64": torch.float64, "bf16": torch.float32}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(shape, dtype, gen):
    """N(0, 1) values in the library's layout (first index fastest)."""
    t = torch.randn(tuple(reversed(shape)), dtype=dtype, device="cuda", generator=gen)
    return t.permute(*reversed(range(len(shape))))


def _uniform(shape, dtype, lo, hi, gen):
    t = torch.rand(tuple(reversed(shape)), dtype=dtype, device="cuda", generator=gen) * (hi - lo) + lo
    return t.permute(*reversed(range(len(shape))))


def _tuple(case, key):
    return tuple(case["%s%d" % (key, k)] for k in range(case["nin"]))


def _orders(case):
    nin = case["nin"]
    got = [(0,) * nin]
    if case["orders"] == "gradient":
        got += [tuple(1 if k == j else 0 for k in range(nin)) for j in range(nin)]
    return got


def _grid_inputs(case, seed):
    gen, dt = _gen(seed), _DT[case["dtype"]]
    cp = _normal(_tuple(case, "n") + (case["nout"],), dt, gen)
    if case["dtype"] == "bf16":
        cp = cp.to(torch.bfloat16)
    w = _uniform(_tuple(case, "n"), dt, 0.5, 2.0, gen) if case["nurbs"] else None
    bars = [_normal(_tuple(case, "s") + (case["nout"],), dt, gen) for _ in _orders(case)] \
        if case["way"] != "forward" else []
    return cp, w, bars


def _dims(case):
    m = 1 if case.get("orders") == "gradient" else 0
    return tuple(sg.SplineDimension(n, d, s, max_derivative_order=m, float_type=_DT[case["dtype"]])
                 for n, d, s in zip(_tuple(case, "n"), _tuple(case, "d"), _tuple(case, "s")))


def _box(shape, rng):
    """A random box of about a quarter of the control points, as ranges per dimension."""
    got = []
    for n in shape:
        ln = max(1, int(round(n * 0.25 ** (1.0 / len(shape)))))
        lo = rng.randint(0, n - ln)
        got.append(range(lo, lo + ln))
    return got


def _refined_shapes(case):
    """Control-point grid sizes of the levels: every knot span is bisected per level."""
    got = [_tuple(case, "n")]
    for _ in range(case["levels"]):
        got.append(tuple(2 * n - d for n, d in zip(got[-1], _tuple(case, "d"))))
    return got


def _refined_boxes(case, seed):
    rng = random.Random(int(seed))
    return [_box(shape, rng) for shape in _refined_shapes(case)[1:]]


def _refined_counts(case, seed):
    return [math.prod(_tuple(case, "n"))] + [math.prod(len(r) for r in b) for b in _refined_boxes(case, seed)]


def _refined_inputs(case, seed):
    gen, dt = _gen(seed), _DT[case["dtype"]]
    x = torch.randn(sum(_refined_counts(case, seed)) * case["nout"], dtype=dt, device="cuda", generator=gen)
    y = torch.randn(math.prod(_tuple(case, "s")) * case["nout"], dtype=dt, device="cuda", generator=gen)
    return x, y


def _batch_specs(case):
    """Grid g's sizes: control points 8..128 and samples 64..smax per dimension, one degree of
    1..3, 1 or 3 outputs, times the control-point sets."""
    got = []
    for g in range(case["grids"]):
        rng = random.Random(case["first"] + g)
        got.append({"n": (rng.randint(8, 128), rng.randint(8, 128)), "d": rng.randint(1, 3),
                    "s": (rng.randint(64, case["smax"]), rng.randint(64, case["smax"])),
                    "ch": rng.choice([1, 3]) * case["sets"]})
    return got


def _batch_inputs(case, seed):
    gen = _gen(seed)
    specs = _batch_specs(case)
    cps = [_normal(s["n"] + (s["ch"],), torch.float32, gen) for s in specs]
    bars = [_normal(s["s"] + (s["ch"],), torch.float32, gen) for s in specs]
    return specs, cps, bars


def _fit_target(case, seed):
    """A smooth surface with noise, flat in the library's layout."""
    gen, dt = _gen(seed), _DT[case["dtype"]]
    u = torch.linspace(0, 1, case["s0"], dtype=torch.float64, device="cuda")
    v = torch.linspace(0, 1, case["s1"], dtype=torch.float64, device="cuda")
    k = torch.rand((case["nout"], 2), dtype=torch.float64, device="cuda", generator=gen) * 20 + 5
    z = torch.stack([torch.sin(k[o, 0] * u)[None, :] * torch.cos(k[o, 1] * v)[:, None] for o in range(case["nout"])])
    z = z + 0.05 * torch.randn(z.shape, dtype=torch.float64, device="cuda", generator=gen)
    return z.to(dt).reshape(-1)


def prepare(case, seed):
    kind, dt = case["kind"], _DT[case.get("dtype", "f32")]
    if kind == "grid":
        cp, w, bars = _grid_inputs(case, seed)
        dims = _dims(case)
        if case["nurbs"]:
            g = sg.NURBSGrid(dims, case["nout"])
            g.weights.copy_(w)
        else:
            g = sg.SplineGrid(dims, case["nout"])
        g.plan(cp.dtype)
        shape = tuple(g.eval.shape)
        evals = [sg.arrays.empty(shape, dt) for _ in _orders(case)] if case["way"] != "adjoint" else []
        grads = [sg.arrays.empty(tuple(cp.shape), dt) for _ in bars]
        if case["autograd"]:
            cp = cp.detach().requires_grad_(True)
        return {"case": case, "grid": g, "orders": _orders(case), "cp": cp, "bars": bars, "evals": evals,
                "grads": grads}
    if kind == "refined":
        x, y = _refined_inputs(case, seed)
        g = sg.SplineGrid(_dims(case), case["nout"])
        for box in _refined_boxes(case, seed):
            g = sg.add_default_local_refinement(g)
            sg.activate_local_control_point_range_(g, *box)
        g.plan(dt)
        A = sg.LinearMap(g)
        return {"case": case, "map": A, "x": x, "y": y, "ax": torch.empty_like(y), "aty": torch.empty_like(x)}
    if kind == "batch":
        specs, cps, bars = _batch_inputs(case, seed)
        grids = []
        for s in specs:
            dims = tuple(sg.SplineDimension(s["n"][k], s["d"], s["s"][k]) for k in range(2))
            grids.append(sg.SplineGrid(dims, s["ch"]))
        evals = [g.eval for g in grids]
        grads = [sg.arrays.empty(tuple(c.shape), torch.float32) for c in cps]
        b = sg.GridBatch(grids)
        b.set_arrays(cps, evals, bars, grads)
        return {"case": case, "batch": b, "evals": evals, "grads": grads}
    c = dict(case, nin=2)
    g = sg.SplineGrid(_dims(c), case["nout"])
    solver = sg.LSQRSolver(sg.LinearMap(g), atol=1e-9, btol=1e-9, conlim=1e9, maxiter=case["iterations"])
    return {"case": case, "solver": solver, "b": _fit_target(case, seed)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "grid":
        g, orders, cp = state["grid"], state["orders"], state["cp"]
        if case["autograd"]:
            ev = sg.autograd.evaluate(g, cp)
            grad, = torch.autograd.grad(ev, cp, state["bars"][0])
            return {"eval": ev.detach(), "grad": grad}
        if state["evals"]:
            if len(orders) > 1:
                sg.evaluate_multi_(g, orders, evals=state["evals"], control_points=cp)
            else:
                sg.evaluate_(g, orders[0], control_points=cp, eval=state["evals"][0])
        for o, e, p in zip(orders, state["bars"], state["grads"]):
            sg.evaluate_adjoint_(g, o, control_points=p, eval=e)
        return {"evals": state["evals"], "grads": state["grads"]}
    if kind == "refined":
        state["map"].mul_(state["ax"], state["x"])
        state["map"].rmul_(state["aty"], state["y"])
        return {"ax": state["ax"], "aty": state["aty"]}
    if kind == "batch":
        state["batch"].run(forward=True, adjoint=True)
        return {"evals": state["evals"], "grads": state["grads"]}
    return {"x": state["solver"].solve(state["b"])}


# ------------------------------------------------------------------------------ work
def _pass_flops(n, d, s, ch):
    """Multiply-adds (two operations) of the separable product, axis by axis."""
    f, nin = 0, len(n)
    for k in range(nin):
        f += 2 * (d[k] + 1) * math.prod(s[:k + 1]) * math.prod(n[k + 1:]) * ch
    return f


def work(case):
    kind = case["kind"]
    if kind == "batch":
        by = fl = 0
        for s in _batch_specs(case):
            v, p = math.prod(s["s"]) * s["ch"], math.prod(s["n"]) * s["ch"]
            by += 4 * (2 * v + 2 * p + sum(s["s"]) * (s["d"] + 1))
            fl += 2 * _pass_flops(s["n"], (s["d"],) * 2, s["s"], s["ch"])
        return {"bytes": by, "flops": fl}
    c = case if "nin" in case else dict(case, nin=2)
    n, d, s, nout = _tuple(c, "n"), _tuple(c, "d"), _tuple(c, "s"), case["nout"]
    es = 8 if case["dtype"] == "f64" else 4
    v, p = math.prod(s) * nout, math.prod(n) * nout
    tables = sum(s[k] * (d[k] + 1) for k in range(len(s)))
    if kind == "fit":
        return {"bytes": es * (v + p + tables), "flops": (2 * case["iterations"] + 1) * _pass_flops(n, d, s, nout)}
    if kind == "refined":
        cnt = sum(_refined_counts(case, 0)) * nout
        fine = _refined_shapes(case)[-1]
        return {"bytes": es * (2 * v + 2 * cnt + tables), "flops": 2 * _pass_flops(fine, d, s, nout)}
    no = len(_orders(case))
    fwd, adj = case["way"] != "adjoint", case["way"] != "forward"
    by = es * tables * no
    if fwd:
        by += es * v * no + (2 if case["dtype"] == "bf16" else es) * p + (es * p // nout if case["nurbs"] else 0)
    if adj:
        by += es * (v + p) * no
    ch = nout + (1 if case["nurbs"] else 0)
    return {"bytes": by, "flops": (int(fwd) + int(adj)) * no * _pass_flops(n, d, s, ch)}


# ------------------------------------------------------------------------------ exact
def _knots(n, d, dtype):
    """The clamped uniform knot vector in the grid's type: distinct values."""
    m = n - d
    return (np.arange(m + 1, dtype=np.float64) / m).astype(np.float64 if dtype == "f64" else np.float32)


def _samples(s, dtype):
    p = np.arange(s, dtype=np.float64) / max(s - 1, 1)
    return p.astype(np.float64 if dtype == "f64" else np.float32).astype(np.float64)


def _basis(values, d, t, order=0):
    """(first basis function, [len(t), d + 1] values) of the B-splines on the clamped knots with
    these distinct interior values; order 0 or 1.  Cox-de Boor in 64 bits."""
    kn = np.concatenate([[values[0]] * d, values, [values[-1]] * d]).astype(np.float64)
    n = len(kn) - d - 1
    span = np.clip(np.searchsorted(kn, t, side="right") - 1, d, n - 1)
    N = np.zeros((len(t), d + 1))
    N[:, 0] = 1.0
    for k in range(1, d + 1):
        new = np.zeros_like(N)
        last = order == 1 and k == d  # the derivative: d (N_i / len_i - N_{i+1} / len_{i+1})
        for j in range(k):
            lo, hi = kn[span + 1 + j - k], kn[span + 1 + j]
            f = N[:, j] / (hi - lo)
            if last:
                new[:, j] -= k * f
                new[:, j + 1] += k * f
            else:
                new[:, j] += f * (hi - t)
                new[:, j + 1] += f * (t - lo)
        N = new
    if order == 1 and d == 0:
        N[:] = 0.0
    return torch.from_numpy(span - d).cuda(), torch.from_numpy(N).cuda()


def _forward(bases, x):
    for k, (b, N) in enumerate(bases):
        view = [1] * x.dim()
        view[k] = N.shape[0]
        y = 0
        for i in range(N.shape[1]):
            y = y + x.index_select(k, b + i) * N[:, i].reshape(view)
        x = y
    return x


def _adjoint(bases, sizes, y):
    for k in reversed(range(len(bases))):
        b, N = bases[k]
        view = [1] * y.dim()
        view[k] = N.shape[0]
        shape = list(y.shape)
        shape[k] = sizes[k]
        x = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for i in range(N.shape[1]):
            x.index_add_(k, b + i, y * N[:, i].reshape(view))
        y = x
    return y


def _bases(case, order=None, values=None):
    c = case if "nin" in case else dict(case, nin=2)
    n, d, s = _tuple(c, "n"), _tuple(c, "d"), _tuple(c, "s")
    return [_basis(_knots(n[k], d[k], case["dtype"]) if values is None else values[k], d[k],
                   _samples(s[k], case["dtype"]), order[k] if order else 0) for k in range(len(n))]


def _insertion(values, d):
    """Distinct knot values after bisecting every span, and the dense matrix from the old to the new
    control points (Boehm's knot insertion, one knot at a time, in 64 bits)."""
    mids = values[:-1] + np.diff(values) / values.dtype.type(2)
    kn = np.concatenate([[values[0]] * d, values, [values[-1]] * d]).astype(np.float64)
    A = np.eye(len(kn) - d - 1)
    for t in mids.astype(np.float64):
        sp = int(np.searchsorted(kn, t, side="right")) - 1
        n = len(kn) - d - 1
        i = np.arange(n + 1)
        a = np.ones(n + 1)
        mid = (i > sp - d) & (i <= sp)
        a[mid] = (t - kn[i[mid]]) / (kn[i[mid] + d] - kn[i[mid]])
        a[i > sp] = 0.0
        up, lo = A[np.minimum(i, n - 1)], A[np.maximum(i - 1, 0)]
        A = a[:, None] * up + (1.0 - a)[:, None] * lo
        kn = np.insert(kn, sp + 1, t)
    new = np.sort(np.concatenate([values, mids]))
    return new, torch.from_numpy(A).cuda()


def _apply(A, k, x):
    return torch.movedim(torch.tensordot(A, x, dims=([1], [k])), 0, k)


def _exact_refined(case, seed):
    x, y = (t.double() for t in _refined_inputs(case, seed))
    d, nout, nin = _tuple(case, "d"), case["nout"], case["nin"]
    shapes, boxes, counts = _refined_shapes(case), _refined_boxes(case, seed), _refined_counts(case, seed)
    values = [_knots(n, dk, case["dtype"]) for n, dk in zip(shapes[0], d)]
    mats = []
    for _ in boxes:
        step = [_insertion(values[k], d[k]) for k in range(nin)]
        values = [s[0] for s in step]
        mats.append([s[1] for s in step])
    col = lambda flat, shape: flat.reshape(tuple(reversed(shape))).permute(*reversed(range(len(shape))))  # noqa: E731
    flat = lambda t: t.permute(*reversed(range(t.dim()))).reshape(-1)  # noqa: E731
    cut = lambda b: tuple(slice(r.start, r.stop) for r in b)  # noqa: E731
    rows = torch.split(x.reshape(nout, -1), counts, dim=1)  # [nout, points of the level]
    cp = col(rows[0].reshape(-1), shapes[0] + (nout,))
    for lev, box in enumerate(boxes):
        for k in range(nin):
            cp = _apply(mats[lev][k], k, cp)
        cp = cp.clone()
        cp[cut(box)] = col(rows[lev + 1].reshape(-1), tuple(len(r) for r in box) + (nout,))
    bases = _bases(case, values=values)
    ax = flat(_forward(bases, cp))
    g = _adjoint(bases, shapes[-1], col(y, _tuple(case, "s") + (nout,)))
    got = []
    for lev in reversed(range(len(boxes))):
        box = cut(boxes[lev])
        got.append(flat(g[box]).reshape(nout, -1))
        g = g.clone()
        g[box] = 0.0
        for k in range(nin):
            g = _apply(mats[lev][k].T.contiguous(), k, g)
    got.append(flat(g).reshape(nout, -1))
    return {"ax": ax, "aty": torch.cat(got[::-1], dim=1).reshape(-1)}


def _exact_fit(case, seed):
    """The same number of LSQR steps (Paige and Saunders, 1982) in 64 bits."""
    b = _fit_target(case, seed).double()
    bases, n, s, nout = _bases(case), (case["n0"], case["n1"]), (case["s0"], case["s1"]), case["nout"]
    col = lambda t, sh: t.reshape((nout,) + sh[::-1]).permute(2, 1, 0)  # noqa: E731
    fwd = lambda v: _forward(bases, col(v, n)).permute(2, 1, 0).reshape(-1)  # noqa: E731
    adj = lambda u: _adjoint(bases, n, col(u, s)).permute(2, 1, 0).reshape(-1)  # noqa: E731
    beta = b.norm()
    u = b / beta
    v = adj(u)
    alpha = v.norm()
    v = v / alpha
    w, x, phibar, rhobar = v.clone(), torch.zeros_like(v), beta, alpha
    for _ in range(case["iterations"]):
        u = fwd(v) - alpha * u
        beta = u.norm()
        u = u / beta
        v = adj(u) - beta * v
        alpha = v.norm()
        v = v / alpha
        rho = torch.hypot(rhobar, beta)
        c, sn = rhobar / rho, beta / rho
        theta, rhobar, phi, phibar = sn * alpha, -c * alpha, c * phibar, sn * phibar
        x = x + (phi / rho) * w
        w = v - (theta / rho) * w
    return {"x": x}


def exact(case, seed):
    kind = case["kind"]
    if kind == "refined":
        return _exact_refined(case, seed)
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "batch":
        specs, cps, bars = _batch_inputs(case, seed)
        evals, grads = [], []
        for s, cp, bar in zip(specs, cps, bars):
            bases = [_basis(_knots(s["n"][k], s["d"], "f32"), s["d"], _samples(s["s"][k], "f32")) for k in range(2)]
            evals.append(_forward(bases, cp.double()))
            grads.append(_adjoint(bases, s["n"], bar.double()))
        return {"evals": evals, "grads": grads}
    cp, w, bars = _grid_inputs(case, seed)
    cp = cp.double()
    evals, grads = [], []
    for i, o in enumerate(_orders(case)):
        bases = _bases(case, o)
        if case["way"] != "adjoint":
            if case["nurbs"]:
                w64 = w.double().unsqueeze(-1)
                evals.append(_forward(bases, cp * w64) / _forward(bases, w64))
            else:
                evals.append(_forward(bases, cp))
        if bars:
            grads.append(_adjoint(bases, _tuple(case, "n"), bars[i].double()))
    if case["autograd"]:
        return {"eval": evals[0], "grad": grads[0]}
    return {"evals": evals, "grads": grads}
