"""The one-lane-per-line cell kernels at the edges of their blocks: cell counts around one block of
every shape (1 to 33 cells in a row, so the last block is ragged), ranges of cells that start inside
the mesh, without Dirichlet DoFs and with them on one face, against the CPU oracle (FP64 to 1e-12,
FP32 to 2e-5 relative in the max norm, the bounds of the operator tests)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TOL = {pmg.F64: 1e-12, pmg.F32: 2e-5}
GEOMETRIES = {
    "full": (1, pmg.GEOMETRY_FULL, pmg.COEFF_NONE),
    "affine": (0, pmg.GEOMETRY_AFFINE, pmg.COEFF_NONE),
    "kappa": (0, pmg.GEOMETRY_AFFINE, pmg.COEFF_KAPPA),
    "invjac": (1, pmg.GEOMETRY_INVJAC, pmg.COEFF_NONE),
}


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("geometry", list(GEOMETRIES))
def test_ragged_blocks_match_oracle(oracle, geometry, degree, dtype):
    deform, geo, coeff = GEOMETRIES[geometry]
    td = torch.float64 if dtype == pmg.F64 else torch.float32
    for n in (1, 2, 3, 5, 8, 9, 15, 33):
        for mask in (0, 1):
            kw = dict(coarse=(n, 1, 1), refine=0, hi=(1.0, 0.25, 0.5), deform=deform, amp=0.1, dirichlet_mask=mask)
            ob = oracle.Box.make(**kw)
            plain, cons, idx = oracle.dofs(ob, degree)
            op = pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(**kw)), degree, dtype, geo, coeff)
            src = np.random.default_rng(n).uniform(-1.0, 1.0, op.m()).astype(np.float64 if dtype == pmg.F64 else np.float32)
            s = torch.tensor(src, dtype=td, device="cuda")
            d = torch.full_like(s, 3.0)  # overwritten
            op.vmult(d, s)

            def reference(first):
                if geometry == "invjac":
                    iJ, jxw = oracle.invjac(ob, degree, coeff)
                    return oracle.vmult_invjac(degree, idx[first:],
                                               np.ascontiguousarray(iJ.reshape(n, -1)[first:]).reshape(-1),
                                               np.ascontiguousarray(jxw.reshape(n, -1)[first:]).reshape(-1), cons,
                                               src.astype(np.float64))
                G = oracle.geometry_G(ob, degree, coeff_kind=coeff).reshape(n, -1)
                return oracle.vmult(degree, idx[first:], G[first:], cons, src.astype(np.float64))

            assert rel_err(d.double().cpu().numpy(), reference(0)) < TOL[dtype], (n, mask)
            first = op.cells_per_group()
            if first < n:  # the cells from the second group on
                op.vmult_cells(d, s, first, n, True)
                assert rel_err(d.double().cpu().numpy(), reference(first)) < TOL[dtype], (n, mask)
