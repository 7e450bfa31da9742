"""What a smoother keeps from call to call (its product vector is zero between calls) after calls that
failed half-way, on vectors with infinities and NaN, with two smoothers on one operator in turn, and on
streams other than the one it was created beside.  Every application is compared with the same one of a
smoother of its own (FP64: 1e-12 relative in the max norm, the operator's bound; the order of its atomic
additions differs from call to call)."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float((a - b).abs().max() / b.abs().max())


def vector(op, seed=1):
    return torch.rand(op.m(), device="cuda", dtype=op.torch_dtype, generator=torch.Generator("cuda").manual_seed(seed)) - 0.5


def smoothed(op, src, degree=4):
    """src smoothed from zero and once more by a new smoother."""
    s, d = pmg.Chebyshev(op, degree), torch.empty_like(src)
    s.estimate()
    s.vmult(d, src)
    s.step(d, src)
    return d


def refused_dot(x):
    """A call that CUDA refuses: it waits for a stream that is being captured."""
    rt = ctypes.CDLL("libcudart.so.12")
    pmg.vector_dot(x, x)
    side, graph = torch.cuda.Stream(), ctypes.c_void_p()
    torch.cuda.synchronize()
    handle = ctypes.c_void_p(side.cuda_stream)
    assert rt.cudaStreamBeginCapture(handle, 1) == 0  # thread-local mode
    with torch.cuda.stream(side):
        with pytest.raises(pmg.PmgError):
            pmg.vector_dot(x, x)
    assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) != 0
    rt.cudaGetLastError()


@pytest.mark.parametrize("degree", [1, 3])
def test_a_call_that_failed_leaves_nothing_behind(monkeypatch, degree):
    monkeypatch.setenv("PMG_DG_FUSE", "0")  # cell and face terms in launches of their own
    op = pmg.DGLaplaceOperator(pmg.Mesh(pmg.Box.make(refine=2)), degree, pmg.F64, 2.0 * (degree + 1) ** 2)
    src = vector(op)
    want = smoothed(op, src)
    s, d = pmg.Chebyshev(op, 4), torch.empty_like(src)
    s.estimate()
    refused_dot(src)
    try:  # whether the refused call's error shows up between the two launches or not,
        s.vmult(d, src)
    except pmg.PmgError:
        pass
    s.vmult(d, src)  # the next call starts from a product of zero
    s.step(d, src)
    assert rel_err(d, want) < 1e-12


@pytest.mark.parametrize("kind", ["patches", "cells", "dg"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_infinities_do_not_stay(kind, bad):
    if kind == "dg":
        op = pmg.DGLaplaceOperator(pmg.Mesh(pmg.Box.make(refine=2)), 2, pmg.F64, 18.0)
    else:
        op = pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(refine=5 if kind == "patches" else 2)), 4, pmg.F64)
    src = vector(op)
    want = smoothed(op, src)
    s, d = pmg.Chebyshev(op, 4), torch.empty_like(src)
    s.estimate()
    broken = src.clone()
    broken[op.m() // 2] = bad
    s.vmult(d, broken)
    s.step(d, broken)
    assert not bool(torch.isfinite(d).all())
    s.vmult(d, src)
    s.step(d, src)
    assert rel_err(d, want) < 1e-12


def test_two_smoothers_on_one_operator():
    op = pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(coarse=(2, 1, 3), refine=2, deform=1)), 3, pmg.F64, pmg.GEOMETRY_FULL)
    src = vector(op)
    degrees = (3, 6)
    want = [smoothed(op, src, k) for k in degrees]
    both = [pmg.Chebyshev(op, k) for k in degrees]
    out = [torch.empty_like(src) for _ in degrees]
    for s in both:
        s.estimate()
    for _ in range(2):
        for s, d in zip(both, out):
            s.vmult(d, src)
        for s, d in zip(both, out):
            s.step(d, src)
        for d, w in zip(out, want):
            assert rel_err(d, w) < 1e-12
