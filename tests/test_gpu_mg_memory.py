"""Device memory of a V-cycle object: the defect and the correction of every level, and a residual only
where the restriction does not take it itself."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu


def test_two_vectors_per_level():
    h = pmg.Hierarchy(pmg.Box.make(refine=5), [4, 2, 1], mg_dtype=pmg.F64, cheb_degree=3)
    h.estimate()
    b = h.fine64.assemble_rhs(0)
    h.mg.vmult(torch.empty_like(b), b)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    mg = pmg.VCycleMultigrid(h.levels, h.transfers, h.smoothers)
    used = free - torch.cuda.mem_get_info()[0]
    vectors = sum(8 * op.m() for op in h.levels)
    assert 0 < used < 3 * vectors
    del mg
