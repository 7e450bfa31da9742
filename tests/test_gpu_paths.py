"""Which kernels a call takes, from the shape of the launches and the labels of the timing registry, where
the results alone cannot tell: patches of cells or single cells, the coarse levels of a V-cycle in one
kernel or in launches of their own, restrictions with or without a pass for the residual; and the kernels
that loop over groups of cells or tiles, with two or more for every warp or block, against the oracle
(FP64 to 1e-12, FP32 to 2e-5 relative in the max norm)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TOL = {pmg.F64: 1e-12, pmg.F32: 2e-5}
PATCHES_PER_BLOCK = {2: 5, 3: 5, 4: 1, 5: 1, 6: 1}


def up(a, b):
    return -(-a // b)


def rel_err(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def apply(op, src):
    d = op.initialize_dof_vector()
    op.vmult(d, torch.as_tensor(src, device="cuda").to(op.torch_dtype))
    return d.double().cpu().numpy()


# ---- loops: two or more groups per warp ----
@pytest.fixture(scope="module")
def looping(oracle):
    out = {}
    for name, degree, deform, geometry, coeff in (("q1_full", 1, 1, pmg.GEOMETRY_FULL, pmg.COEFF_NONE),
                                                  ("q1_invjac", 1, 1, pmg.GEOMETRY_INVJAC, pmg.COEFF_NONE),
                                                  ("q2_kappa", 2, 0, pmg.GEOMETRY_AFFINE, pmg.COEFF_KAPPA)):
        box = pmg.Box.make(refine=6, deform=deform)
        ob = oracle.Box.make(refine=6, deform=deform, amp=box.amp)
        plain, cons, idx = oracle.dofs(ob, degree)
        src = np.random.default_rng(degree).uniform(-1.0, 1.0, cons.shape[0])
        if geometry == pmg.GEOMETRY_INVJAC:
            ref = oracle.vmult_invjac(degree, idx, *oracle.invjac(ob, degree, coeff), cons, src)
        else:
            ref = oracle.vmult(degree, idx, oracle.geometry_G(ob, degree, coeff_kind=coeff), cons, src)
        out[name] = (box, degree, geometry, coeff, src, ref)
    return out


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("case", ["q1_full", "q1_invjac", "q2_kappa"])
def test_slab_kernels_take_two_groups_per_warp(looping, case, dtype):
    box, degree, geometry, coeff, src, ref = looping[case]
    op = pmg.LaplaceOperator(pmg.Mesh(box), degree, dtype, geometry, coeff)
    for _ in range(2):
        assert rel_err(apply(op, src), ref) < TOL[dtype]
        groups, warps = op.last_launch()
        assert groups == up(op.n_cells(), 32 // (degree + 1)) and groups >= 2 * warps > 0


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
def test_dg_tiles_take_two_per_block(monkeypatch, dtype):
    op = pmg.DGLaplaceOperator(pmg.Mesh(pmg.Box.make(refine=6)), 3, dtype, 32.0)
    src = np.random.default_rng(3).uniform(-1.0, 1.0, op.m())
    by_lines = apply(op, src)
    for kernel in (pmg.KERNEL_VMULT_CELL, pmg.KERNEL_DG_FACES):
        assert op.last_launch(kernel) == (op.n_cells(), up(op.n_cells(), 8))
    monkeypatch.setenv("PMG_DG_FACE", "2")
    by_tiles = apply(op, src)
    for kernel in (pmg.KERNEL_VMULT_CELL, pmg.KERNEL_DG_FACES):
        tiles, blocks = op.last_launch(kernel)
        assert tiles == op.n_cells() // 64 and tiles >= 2 * blocks > 0
    assert rel_err(by_tiles, by_lines) < TOL[dtype]


# ---- patches ----
@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("degree", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("coarse,refine,taken", [((2, 1, 1), 5, True), ((3, 2, 1), 5, True), ((1, 1, 1), 3, False),
                                                 ((64, 32, 32), 0, False)])
def test_patches_where_they_fill_the_device(coarse, refine, taken, degree, dtype):
    op = pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(coarse=coarse, refine=refine)), degree, dtype)
    s, d = op.initialize_dof_vector(), op.initialize_dof_vector()
    op.vmult_cells(d, s, 0, op.n_cells(), True)
    cells, by_cells = op.last_launch()
    op.vmult(d, s)
    again, blocks = op.last_launch()
    assert cells == again == op.n_cells()
    by_patches = up(op.n_cells() // 8, PATCHES_PER_BLOCK[degree])
    # (FP32 Q4 has four pairs of cells to a block, as many cells as a patch: nothing to tell them apart)
    assert (by_cells == by_patches) == (degree == 4 and dtype == pmg.F32)
    assert blocks == (by_patches if taken else by_cells)


# ---- V-cycles ----
def launches(h, labels):
    """How often each label occurs in one V-cycle."""
    b = h.levels[-1].assemble_rhs(0)
    x = torch.empty_like(b)
    h.estimate()
    pmg.profile_enable(True)
    try:
        pmg.profile_reset()
        h.mg.vmult(x, b)
        torch.cuda.synchronize()
        return [pmg.profile_query(k)[1] for k in labels]
    finally:
        pmg.profile_reset()
        pmg.profile_enable(False)


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("pseq,h_degree,coarse,refine,kw,tail", [
    ([4, 2, 1], 1, (1, 1, 1), 5, {}, 4),                                                # 8 to 729 DoFs in the kernel
    ([1], 1, (3, 3, 3), 3, dict(coeff_kind=pmg.COEFF_KAPPA), 2),                        # 64 and 343
    ([1], 1, (1, 1, 1), 4, dict(geometry=pmg.GEOMETRY_FULL), 4),
    ([2], 2, (1, 1, 1), 3, {}, 3),                                                      # 27 to 729, degree 2
    ([2], 2, (1, 1, 1), 3, dict(coeff_kind=pmg.COEFF_KAPPA), 0),                        # not with a coefficient
    ([3], 3, (1, 1, 1), 2, {}, 0), ([1], 1, (1, 1, 1), 2, {}, 3),                       # another degree; all levels
    ([3, 1], 1, (1, 1, 1), 3, dict(dg=True), 4)])
def test_cycle_launches(pseq, h_degree, coarse, refine, kw, tail, dtype):
    box = pmg.Box.make(coarse=coarse, refine=refine, deform=1 if "geometry" in kw else 0)
    cheb = 3
    h = pmg.Hierarchy(box, pseq, mg_dtype=dtype, cheb_degree=cheb, h_degree=h_degree, **kw)
    tails, up_, down, updates = launches(h, ["mg_tail", "transfer_prolongate", "transfer_restrict", "vector_update"])
    levels = len(h.levels)
    assert tails == (1 if tail else 0)
    assert up_ == down == levels - max(tail, 1)
    # the conversions in and out; from zero and onwards `cheb` updates each; level 0 by its own degree
    want = 2 + 2 * cheb * (levels - max(tail, 1)) + (0 if tail else h.smoothers[0].info()["degree"])
    if kw.get("dg"):  # all but the first of both run in the DG kernel, and its restriction needs the residual
        want += 1 - 2 * (cheb - 1)
    assert updates == want
