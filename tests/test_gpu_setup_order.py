"""Objects are ready for any stream when their creation returns: streams that do not wait for the default
one (torch's side streams) may use them at once.  The results are compared with those of objects made and
used on the default stream (FP64: 1e-12 relative in the max norm, the operator's bound)."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float((a - b).abs().max() / b.abs().max())


def busy():
    """About 0.1 s of work on the default stream."""
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)
    assert not torch.cuda.default_stream().query()


def test_smoother_of_an_operator_that_has_its_diagonal():
    op = pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(refine=3)), 2, pmg.F64)
    op.compute_diagonal()
    src = torch.rand(op.m(), device="cuda", dtype=torch.float64)

    def run(s):
        d = torch.empty_like(src)
        s.estimate()
        s.vmult(d, src)
        s.step(d, src)
        return d

    want = run(pmg.Chebyshev(op, 4))
    side = torch.cuda.Stream()
    busy()
    s = pmg.Chebyshev(op, 4)
    assert torch.cuda.default_stream().query()
    with torch.cuda.stream(side):
        got = run(s)
    torch.cuda.synchronize()
    assert rel_err(got, want) < 1e-12


def test_multigrid_on_a_side_stream():
    def hierarchy():
        return pmg.Hierarchy(pmg.Box.make(refine=3), [3, 1], mg_dtype=pmg.F64, cheb_degree=3)

    def run(h, b):
        x = torch.zeros_like(b)
        h.estimate()
        h.mg.vmult(x, b)
        h.mg.vmult(x, b)  # (from the captured graph)
        y, info = h.solve(b, reduce=1e-10)
        return x, y, info["iterations"]

    first = hierarchy()
    b = first.fine64.assemble_rhs(0)
    want = run(first, b)
    side = torch.cuda.Stream()
    busy()
    h = hierarchy()
    assert torch.cuda.default_stream().query()
    with torch.cuda.stream(side):
        got = run(h, b)
    torch.cuda.synchronize()
    assert got[2] == want[2]
    # a cycle chains some hundred vector operations of the operator's accuracy; the solve stops at 1e-10
    assert rel_err(got[0], want[0]) < 1e-10 and rel_err(got[1], want[1]) < 1e-9
