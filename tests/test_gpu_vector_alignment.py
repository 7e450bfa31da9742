"""Vector entry points on vectors whose start is not 16-byte aligned and whose length is no multiple
of the wide access (the one-entry-per-thread forms), against torch in the same precision: bounds of a
few roundings per entry, 1e-14 / 1e-6 relative to the largest entry."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 1e-14, torch.float32: 1e-6}


def vectors(n, dtype, offset, count):
    g = torch.Generator(device="cuda").manual_seed(n + offset)
    return [(torch.rand(n + 8, generator=g, device="cuda", dtype=torch.float64) - 0.5).to(dtype)[offset:offset + n]
            for _ in range(count)]


def close(a, b):
    assert float((a.double() - b.double()).abs().max()) <= TOL[a.dtype] * max(1.0, float(b.double().abs().max()))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 2, 5, 1023, 4099])
def test_vector_entry_points(n, offset, dtype):
    a, b, c, d, e, out = vectors(n, dtype, offset, 6)
    y = b.clone()[:]
    w = vectors(n, dtype, offset, 1)[0]
    w.copy_(b)
    pmg.vector_axpy(w, a, 0.75)
    close(w, y + 0.75 * a)
    w.copy_(b)
    pmg.vector_xpay(w, a, -0.5)
    close(w, a - 0.5 * y)
    pmg.vector_pointwise_mult(out, a, b)
    close(out, a * b)
    pmg.vector_chebyshev_step(out, a, None, b, c, d, 0.3, 0.7)
    close(out, a + 0.3 * a + 0.7 * d * (b - c))
    w.copy_(e)
    pmg.vector_chebyshev_step(w, a, w, b, c, d, 0.3, 0.7)
    close(w, a + 0.3 * (a - e) + 0.7 * d * (b - c))
    other = torch.float32 if dtype == torch.float64 else torch.float64
    z = vectors(n, other, offset, 1)[0]
    pmg.vector_copy(z, a)
    assert torch.equal(z, a.to(other))
    ref = float(torch.dot(a.double(), b.double()))
    assert abs(pmg.vector_dot(a, b) - ref) <= 1e-13 * max(1.0, float(torch.dot(a.double().abs(), b.double().abs())))


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
def test_vmult_and_smoother_on_unaligned_vectors(dtype):
    op = pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(coarse=(3, 2, 1), refine=1)), 3, dtype)
    td = torch.float64 if dtype == pmg.F64 else torch.float32
    n = op.m()
    src = vectors(n, td, 1, 1)[0]
    ref, got = op.initialize_dof_vector(), vectors(n, td, 1, 1)[0]
    op.vmult(ref, src.clone())
    op.vmult(got, src)
    assert float((got - ref).abs().max()) <= (1e-14 if dtype == pmg.F64 else 1e-6) * float(ref.abs().max())
    s = pmg.Chebyshev(op, 4)
    for f in (s.vmult, s.step):
        f(ref, src.clone())
        f(got, src)
        assert float((got - ref).abs().max()) <= (1e-12 if dtype == pmg.F64 else 1e-5) * float(ref.abs().max())
