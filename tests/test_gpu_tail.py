"""The one-kernel coarse levels of a V-cycle against the same cycle put together from the public
smoothers, operators and transfers level by level: hierarchies whose levels all fit into one block's
shared memory and hierarchies whose upper levels run in launches of their own; degree 1 with
every geometry, degree 2 plain; odd and even Chebyshev degrees (FP64 to 1e-11, FP32 to 1e-4 relative
in the max norm: a cycle chains some hundred vector operations of the operator's accuracy)."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TOL = {pmg.F64: 1e-11, pmg.F32: 1e-4}
GEOMETRIES = {
    "affine": (0, pmg.GEOMETRY_AFFINE, pmg.COEFF_NONE),
    "kappa": (0, pmg.GEOMETRY_AFFINE, pmg.COEFF_KAPPA),
    "full": (1, pmg.GEOMETRY_FULL, pmg.COEFF_NONE),
}


def vcycle(h, defect):
    """One V-cycle on the levels' own objects."""
    top = len(h.levels) - 1

    def level(l, d):
        x = torch.empty_like(d)
        h.smoothers[l].vmult(x, d)
        if l == 0:
            return x
        r = torch.empty_like(d)
        h.levels[l].vmult(r, x)
        r = d - r
        dc = h.levels[l - 1].initialize_dof_vector()
        h.transfers[l].restrict_and_add(dc, r)
        h.transfers[l].prolongate_and_add(x, level(l - 1, dc))
        h.smoothers[l].step(x, d)
        return x

    return level(top, defect)


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("geometry,degree,coarse,refine,cheb",
                         [("affine", 1, (1, 1, 1), 1, 2), ("affine", 1, (1, 1, 1), 3, 5), ("affine", 1, (2, 1, 3), 4, 4),
                          ("affine", 2, (1, 1, 1), 2, 3), ("affine", 2, (2, 2, 2), 3, 3), ("affine", 1, (3, 3, 3), 4, 1),
                          ("kappa", 1, (3, 3, 3), 3, 4), ("kappa", 1, (1, 2, 1), 2, 3), ("full", 1, (1, 1, 1), 4, 3),
                          ("full", 1, (3, 1, 2), 2, 4)])
def test_vcycle_matches_its_parts(geometry, degree, coarse, refine, cheb, dtype):
    deform, geo, coeff = GEOMETRIES[geometry]
    box = pmg.Box.make(coarse=coarse, refine=refine, deform=deform, amp=0.1)
    h = pmg.Hierarchy(box, [degree], mg_dtype=dtype, cheb_degree=cheb, geometry=geo, coeff_kind=coeff, h_degree=degree)
    h.estimate()
    d = h.levels[-1].assemble_rhs(0)
    d = d * (1.0 + 0.5 * torch.rand_like(d))
    want = vcycle(h, d)
    x = torch.empty_like(d)
    for _ in range(2):  # the second cycle finds what the first left in the levels' vectors
        h.mg.vmult(x, d)
        err = float((x - want).abs().max() / want.abs().max())
        assert err < TOL[dtype]
