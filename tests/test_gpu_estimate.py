"""The smoother's eigenvalue estimate against the same conjugate gradient (Lanczos) run from the public
operator and diagonal in torch: definite and indefinite operators (a DG penalty below the one that makes
the form positive), fewer and more iterations than the host looks at together; and an operator with a
negative coefficient, whose Jacobi-preconditioned spectrum is that of the positive one.  Perturbing the
products by 1e-15 moves the Ritz values of these cases by at most 1e-12 of the largest: 1e-9 for the
products' rounding."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu


def lanczos(op, iterations):
    """(smallest, largest Ritz value, how often p.Ap < 0) of the run the estimate makes."""
    inv = op.get_matrix_diagonal_inverse()
    assert float(inv.min()) > 0
    r = torch.arange(op.m(), device="cuda").remainder(11).double()
    r = r - r.mean()
    z = inv * r
    p, v, rho, alpha, beta, carry, negative = z, torch.empty_like(z), float(r @ z), 0.0, 0.0, 0.0, 0
    diag, off = [], []
    for it in range(1, iterations + 1):
        if it > 1:
            p = z + beta * p
        op.vmult(v, p)
        pv = float(p @ v)
        negative += pv < 0
        previous, alpha = alpha, rho / pv
        if it > 1:
            diag.append(1.0 / previous + carry)
            carry = beta / previous
            off.append(math.sqrt(beta) / previous)
        r = r - alpha * v
        z = inv * r
        old, rho = rho, float(r @ z)
        beta = rho / old
    ev = np.linalg.eigvalsh(np.diag(diag) + np.diag(off[:-1], 1) + np.diag(off[:-1], -1))
    return ev[0], ev[-1], negative


@pytest.mark.parametrize("degree,penalty,iterations", [(p, c, n) for p, c in ((1, 0.7), (2, 2.5), (3, 5.0), (2, 8.0))
                                                       for n in (10, 16, 17)] + [(2, 2.5, 40), (2, 8.0, 40)])
def test_estimate_matches_lanczos(degree, penalty, iterations):
    box = pmg.Box.make(coarse=(2, 1, 1), refine=1, hi=(2.0, 1.0, 1.0))
    op = pmg.DGLaplaceOperator(pmg.Mesh(box), degree, pmg.F64, penalty)
    smoother = pmg.Chebyshev(op, 5, 15.0, iterations)
    low, high, negative = lanczos(op, iterations)
    assert (negative > 0) == (penalty < 8.0)
    for _ in range(2):  # (a second estimate keeps its work vectors)
        smoother.estimate()
        info = smoother.info()
        assert info["cg_iterations"] == iterations
        assert abs(info["max_eigenvalue"] - 1.2 * high) < 1e-9 * high
        assert abs(info["min_eigenvalue"] - low) < 1e-9 * high


@pytest.mark.parametrize("dtype,tol", [(pmg.F64, 1e-9), (pmg.F32, 1e-3)])
@pytest.mark.parametrize("degree", [1, 2, 4])
def test_estimate_of_a_negative_operator(degree, dtype, tol):
    mesh = pmg.Mesh(pmg.Box.make(coarse=(3, 2, 1), refine=1, dirichlet_mask=0))
    found = []
    for sign in (1.0, -1.0):
        values = np.full((mesh.n_cells(), (degree + 1) ** 3), 1.5 * sign)
        op = pmg.LaplaceOperator(mesh, degree, dtype, pmg.GEOMETRY_AFFINE, pmg.COEFF_VALUES, values)
        smoother = pmg.Chebyshev(op, 4, 15.0, 10)
        smoother.estimate()
        found.append(smoother.info())
    for key in ("min_eigenvalue", "max_eigenvalue"):
        assert abs(found[1][key] - found[0][key]) < tol * found[0]["max_eigenvalue"]
