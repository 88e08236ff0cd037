"""A large 2D grid's adjoint runs as two passes through an intermediate of its plan: calls on
several streams, tuning beside them and captures keep each result apart."""
import pytest

pytestmark = pytest.mark.gpu

N, NS, NOUT = (96, 80), (2048, 1024), 1


def _large(sg):
    """A grid whose adjoint goes through the plan's intermediate, its cotangent and gradient."""
    import torch
    g = sg.SplineGrid(tuple(sg.SplineDimension(n, 3, s) for n, s in zip(N, NS)), NOUT)
    gen = torch.Generator().manual_seed(11)
    cot = sg.arrays.from_any(torch.randn(NS + (NOUT,), generator=gen), torch.float32)
    want = sg.arrays.empty(N + (NOUT,), torch.float32)
    sg.evaluate_adjoint_(g, eval=cot, control_points=want)
    torch.cuda.synchronize()
    assert g.plan(torch.float32).paths() == ("fused", "separable")
    return g, cot, want


def test_tuning_waits_for_another_streams_adjoints(sg):
    """sg_grid_plan_tune writes the intermediate that adjoints still queued on another stream read."""
    import torch
    g, cot, want = _large(sg)
    queued = [sg.arrays.zeros(N + (NOUT,), torch.float32) for _ in range(40)]
    other = sg.arrays.from_any(-cot, torch.float32)
    scratch = sg.arrays.empty(N + (NOUT,), torch.float32)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(2_000_000)  # the calls below are queued before any of them runs
        for q in queued:
            sg.evaluate_adjoint_(g, eval=cot, control_points=q)
    with torch.cuda.stream(b):
        sg.tune_adjoint_(g, eval=other, control_points=scratch)
    torch.cuda.synchronize()
    for q in queued:
        assert torch.equal(q, want)
    # and adjoints that follow the tuning, on the first stream
    with torch.cuda.stream(a):
        queued[0].zero_()
        sg.evaluate_adjoint_(g, eval=cot, control_points=queued[0])
    torch.cuda.synchronize()
    assert torch.equal(queued[0], want)
    g.plan(torch.float32).untune()


@pytest.mark.parametrize("busy", [False, True])
def test_another_threads_capture_survives_the_adjoint(sg, busy):
    """An adjoint on a second stream asks whether the first one's is done; asking must neither fail
    nor end a capture (torch's default, global mode) that another thread has under way."""
    import threading

    import torch
    g, cot, want = _large(sg)
    got = sg.arrays.zeros(N + (NOUT,), torch.float32)
    first = sg.arrays.zeros(N + (NOUT,), torch.float32)
    a, b, s = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(1000, device="cuda")
    with torch.cuda.stream(b):
        x.add_(0)  # the streams exist before the capture
    torch.cuda.synchronize()
    errors = []

    def on_b():
        try:
            with torch.cuda.stream(b):
                sg.evaluate_adjoint_(g, eval=cot, control_points=got)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    with torch.cuda.stream(a):
        if busy:
            torch.cuda._sleep(20_000_000)
        sg.evaluate_adjoint_(g, eval=cot, control_points=first)
    if not busy:
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        graph.capture_begin(capture_error_mode="global")
        x.add_(1)
        t = threading.Thread(target=on_b)
        t.start()
        t.join()
        x.add_(1)
        graph.capture_end()
    assert not errors, errors
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(first, want)
    assert float(x[0]) == 2.0 and float(x[-1]) == 2.0
