"""The kernel on patches of 2 x 2 x 2 cells against the same operator applied cell by cell: every degree
and type, boxes of several coarse cells, all faces, one face and no face constrained, a ragged last block;
and cells in an order without such patches (FP64 to 1e-12, FP32 to 2e-5 relative in the max norm, the
bounds of the operator tests)."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TOL = {pmg.F64: 1e-12, pmg.F32: 2e-5}


def rel_err(a, b):
    return float((a.double() - b.double()).abs().max() / b.double().abs().max())


def random_vector(op, seed=1):
    g = torch.Generator("cuda").manual_seed(seed)
    return torch.rand(op.m(), device="cuda", dtype=op.torch_dtype, generator=g) - 0.5


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("degree", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("coarse,refine,mask", [((1, 1, 1), 5, 0x3f), ((3, 2, 1), 5, 1), ((2, 1, 1), 5, 0)])
def test_patches_match_cells(coarse, refine, mask, degree, dtype):
    box = pmg.Box.make(coarse=coarse, refine=refine, hi=(1.0, 0.5, 2.0), dirichlet_mask=mask)
    op = pmg.LaplaceOperator(pmg.Mesh(box), degree, dtype)
    s = random_vector(op)
    got, want = torch.full_like(s, 3.0), torch.full_like(s, 5.0)  # overwritten
    op.vmult(got, s)
    op.vmult_cells(want, s, 0, op.n_cells(), True)
    assert rel_err(got, want) < TOL[dtype]
    again = torch.empty_like(s)
    op.vmult(again, s)
    assert rel_err(again, got) < TOL[dtype]


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
def test_other_cell_orders(dtype):
    degree = 3
    ops = [pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(coarse=c, refine=r)), degree, dtype)
           for c, r in (((1, 1, 1), 5), ((32, 32, 32), 0))]
    n = 32 * degree + 1
    place = []  # lattice point -> DoF
    for op in ops:
        i, j, k = torch.as_tensor(op.dof_lattice(), dtype=torch.int64).cuda().unbind(1)
        place.append(torch.argsort((k * n + j) * n + i))
    x = random_vector(ops[0])
    out = []
    for op, at in zip(ops, place):
        s, d = torch.empty_like(x), torch.empty_like(x)
        s[at] = x
        op.vmult(d, s)
        out.append(d[at])
    assert rel_err(out[0], out[1]) < TOL[dtype]
