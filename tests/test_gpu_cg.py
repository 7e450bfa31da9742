"""CG iterations against the same iterations put together from the public operator, V-cycle and
diagonal in torch: operator and V-cycle in the same and in different types (the residual and the
direction are converted inside the updates), without a V-cycle, vectors that start on no 16-byte
boundary, odd lengths.  Three iterations chain some dozens of operations of the types' accuracy:
1e-10 where everything is FP64, else 1e-4, relative in the max norm."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TORCH = {pmg.F64: torch.float64, pmg.F32: torch.float32}


def cg(A, precondition, b, iterations):
    x, r = torch.zeros_like(b), b.clone()
    p = v = rho = None
    for _ in range(iterations):
        z = precondition(r)
        old, rho = rho, torch.dot(r.double(), z.double())
        p = z.clone() if p is None else z + (rho / old).to(b.dtype) * p
        v = torch.empty_like(p)
        A.vmult(v, p)
        alpha = (rho / torch.dot(p.double(), v.double())).to(b.dtype)
        x, r = x + alpha * p, r - alpha * v
    return x


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("precond", [None, pmg.F64, pmg.F32])
@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
def test_cg_matches_its_parts(dtype, precond, offset):
    box = pmg.Box.make(coarse=(2, 1, 3), refine=1)
    h = pmg.Hierarchy(box, [3, 1], mg_dtype=pmg.F64 if precond is None else precond)
    A = h.fine64 if dtype == pmg.F64 else pmg.LaplaceOperator(h.meshes[-1], 3, dtype)
    b = A.assemble_rhs(0)
    assert b.numel() % 2 == 1
    b = b * (1.0 + 0.5 * torch.rand(b.numel(), device="cuda", dtype=b.dtype,
                                    generator=torch.Generator("cuda").manual_seed(1)))
    if precond is None:
        A.compute_diagonal()
        inv = A.get_matrix_diagonal_inverse()

        def precondition(r):
            return inv * r
    else:
        def precondition(r):
            z = torch.empty_like(r)
            h.mg.vmult(z, r)
            return z
    tol = 1e-10 if dtype == pmg.F64 and precond != pmg.F32 else 1e-4
    buf = torch.zeros(2, b.numel() + 7, device="cuda", dtype=TORCH[dtype])
    x, rhs = (buf[k][offset:offset + b.numel()] for k in (0, 1))
    rhs.copy_(b)
    for iterations in (1, 3):
        want = cg(A, precondition, b, iterations)
        x.zero_()
        info = pmg.solve_cg(A, x, rhs, None if precond is None else h.mg, reduce=1e-30, abs_tol=0.0,
                            max_iterations=iterations, raise_on_noconv=False)
        assert info["iterations"] == iterations and not info["converged"]
        assert float((x - want).abs().max() / want.abs().max()) < tol
    assert torch.equal(rhs, b)
