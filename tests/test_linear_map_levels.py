"""Copies between a flat vector and the levels of locally refined control points: the vector has
to hold the levels as they are now.  A map made before a level was refined further has another
length; its calls raise, and nothing is copied past the vector's end.  (Host logic: tensors that
claim to be on a GPU, and a library that records the copies.)"""
import types

import pytest
import torch

from splinegrids import linear_map
from splinegrids.control_points import LocallyRefinedControlPoints, LocalRefinement


class _OnGpu(torch.Tensor):
    is_cuda = property(lambda self: True)


def _colmajor(n, nout):
    return torch.arange(float(n * nout)).reshape(nout, n).t().as_subclass(_OnGpu)


def _levels(rows, nout):
    lrs = [LocalRefinement([0], [], torch.zeros((n, 1), dtype=torch.int32), _colmajor(n, nout)) for n in rows]
    return LocallyRefinedControlPoints([torch.zeros((9, nout))] * len(rows), lrs)


@pytest.fixture
def copies(monkeypatch):
    """The byte ranges that copies touch, per call."""
    seen = []

    def copy_list(k, dst, src, nbytes, stream):
        seen.append([(dst[i], src[i], nbytes[i]) for i in range(k)])
        return 0

    fake = types.SimpleNamespace(load=lambda: types.SimpleNamespace(sg_copy_list=copy_list), check=lambda rc: None,
                                 stream_handle=lambda: 0)
    monkeypatch.setattr(linear_map, "_lib", fake)
    return seen


@pytest.mark.parametrize("out", [False, True])
@pytest.mark.parametrize("nout", [1, 3])
def test_copies_cover_the_vector_exactly(copies, nout, out):
    cps = _levels((4, 0, 3), nout)
    x = torch.zeros(7 * nout).as_subclass(_OnGpu)
    linear_map._copy_out(x, cps) if out else linear_map._copy_in(cps, x)
    (call,) = copies
    got = sorted((d if out else s, n) for d, s, n in call)
    assert got[0][0] == x.data_ptr() and sum(n for _, n in got) == 4 * x.numel()
    assert all(a + n == b for (a, n), (b, _) in zip(got, got[1:]))


@pytest.mark.parametrize("out", [False, True])
@pytest.mark.parametrize("length", [0, 9, 20, 22])
def test_a_vector_of_another_length_is_refused(copies, length, out):
    cps = _levels((4, 3), 3)
    x = torch.zeros(length).as_subclass(_OnGpu)
    with pytest.raises((AssertionError, ValueError, RuntimeError)):
        linear_map._copy_out(x, cps) if out else linear_map._copy_in(cps, x)
    assert not copies


@pytest.mark.parametrize("out", [False, True])
def test_values_of_another_shape_than_their_indices_are_refused(copies, out):
    cps = _levels((4, 3), 3)
    cps.local_refinements[0].refinement_values = _colmajor(4, 2)
    x = torch.zeros(21).as_subclass(_OnGpu)
    with pytest.raises((AssertionError, ValueError, RuntimeError)):
        linear_map._copy_out(x, cps) if out else linear_map._copy_in(cps, x)
    assert not copies
