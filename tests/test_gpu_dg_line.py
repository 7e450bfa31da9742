"""The one-lane-per-line DG kernel (the default form) at the edges of its blocks: meshes of 1 to 24
cells without and with every kind of boundary face, vectors off the 16-byte grid, and the Chebyshev
steps taken inside the kernel against the separate vmult and update (PMG_DG_FUSE=0).  FP64 to 1e-12,
FP32 to 2e-5 relative in the max norm against the CPU oracle, as the operator's other tests."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu

TOL = {pmg.F64: 1e-12, pmg.F32: 2e-5}


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 6])
def test_dg_line_kernel_matches_oracle(oracle, p, dtype):
    td = torch.float64 if dtype == pmg.F64 else torch.float32
    for coarse, refine, mask in (((1, 1, 1), 0, 0x3F), ((2, 1, 1), 0, 0x00), ((3, 1, 2), 0, 0x2A), ((1, 3, 1), 1, 0x15)):
        kw = dict(coarse=coarse, refine=refine, hi=(1.0, 0.5, 2.0), dirichlet_mask=mask)
        ob = oracle.Box.make(**kw)
        c_pen = 2.0 * (p + 1) ** 2
        op = pmg.DGLaplaceOperator(pmg.Mesh(pmg.Box.make(**kw)), p, dtype, c_pen)
        src = np.random.default_rng(p).uniform(-1, 1, op.m())
        ref = oracle.dg_vmult(ob, p, c_pen, src)
        for offset in (0, 1):
            s = torch.zeros(op.m() + 2, dtype=td, device="cuda")[offset:offset + op.m()]
            s.copy_(torch.tensor(src, dtype=td))
            d = torch.full((op.m() + 2,), 5.0, dtype=td, device="cuda")[offset:offset + op.m()]
            op.vmult(d, s)
            assert rel_err(d.double().cpu().numpy(), ref) < TOL[dtype], (coarse, refine, mask, offset)


@pytest.mark.parametrize("dtype", [pmg.F64, pmg.F32])
@pytest.mark.parametrize("p", [1, 2, 4, 6])
def test_dg_steps_in_line_kernel(monkeypatch, p, dtype):
    op = pmg.DGLaplaceOperator(pmg.Mesh(pmg.Box.make(coarse=(2, 1, 1), refine=1, dirichlet_mask=0x3C)), p, dtype,
                               2.0 * (p + 1) ** 2)
    td = torch.float64 if dtype == pmg.F64 else torch.float32
    src = torch.tensor(np.random.default_rng(7).uniform(-1, 1, op.m()), dtype=td, device="cuda")
    for degree in (1, 2, 5):
        got = []
        for fuse in (None, "0"):
            if fuse is None:
                monkeypatch.delenv("PMG_DG_FUSE", raising=False)
            else:
                monkeypatch.setenv("PMG_DG_FUSE", fuse)
            sm = pmg.Chebyshev(op, degree=degree)
            sm.estimate()
            d = op.initialize_dof_vector()
            sm.vmult(d, src)
            sm.step(d, src)
            got.append(d.double().cpu().numpy())
        assert rel_err(got[0], got[1]) < (1e-12 if dtype == pmg.F64 else 1e-5)
