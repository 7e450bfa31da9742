"""A V-cycle whose restrictions take the residual themselves against the same cycle put together from the
public smoothers, operators and transfers: p- and h-levels, full geometry, a coefficient, DG on top
(whose transfer keeps the residual's pass), boxes without constrained DoFs on some faces (FP64 to 1e-11,
FP32 to 1e-4 relative in the max norm: a cycle chains some hundred vector operations of the operator's
accuracy)."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TOL = {pmg.F64: 1e-11, pmg.F32: 1e-4}


def vcycle(h, defect):
    """One V-cycle on the levels' own objects."""
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

    return level(len(h.levels) - 1, defect)


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("pseq,h_degree,coarse,refine,kw", [
    ([6, 3, 1], 1, (2, 1, 1), 3, {}),
    ([4, 2, 1], 1, (3, 2, 1), 3, dict(coeff_kind=pmg.COEFF_KAPPA)),
    ([5, 4, 3, 2], 2, (1, 2, 1), 2, dict(geometry=pmg.GEOMETRY_FULL)),
    ([3], 3, (1, 1, 1), 3, {}), ([4], 4, (2, 1, 1), 2, {}), ([2], 2, (1, 1, 2), 4, {}),
    ([3, 1], 1, (1, 1, 1), 3, dict(dg=True))])
@pytest.mark.parametrize("mask", [0x3f, 0x05])
def test_vcycle_matches_its_parts(pseq, h_degree, coarse, refine, kw, mask, dtype):
    if kw.get("dg") and mask != 0x3f:
        pytest.skip("one mask is enough where Dirichlet data is imposed weakly")
    deform = 1 if kw.get("geometry") == pmg.GEOMETRY_FULL else 0
    box = pmg.Box.make(coarse=coarse, refine=refine, deform=deform, amp=0.1, dirichlet_mask=mask)
    h = pmg.Hierarchy(box, pseq, mg_dtype=dtype, cheb_degree=3, h_degree=h_degree, **kw)
    h.estimate()
    d = h.levels[-1].assemble_rhs(0)
    d = d * (1.0 + 0.5 * torch.rand(d.numel(), device="cuda", dtype=d.dtype, generator=torch.Generator("cuda").manual_seed(1)))
    want = vcycle(h, d)
    x = torch.empty_like(d)
    for _ in range(2):  # the second cycle finds what the first left in the levels' vectors
        h.mg.vmult(x, d)
        assert float((x - want).abs().max() / want.abs().max()) < TOL[dtype]
