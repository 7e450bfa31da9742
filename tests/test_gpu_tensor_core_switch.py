"""pmg_operator_set_tensor_cores between two V-cycles takes effect in the next one, which a CUDA graph
replays.  Two TF32 cycles differ from each other by as much as from an FP32 one (an FP32 rounding moves an
entry across a TF32 step), so what is compared is how far a cycle is from the FP32 one: FP32 rounding
(1e-5 in the 2-norm) with the switch off, with it on half to twice as far as a cycle whose levels were
switched before their first cycle."""
import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu


def hierarchy():
    h = pmg.Hierarchy(pmg.Box.make(coarse=(3, 3, 3), refine=2), [6, 3, 1], mg_dtype=pmg.F32, cheb_degree=4,
                      coeff_kind=pmg.COEFF_KAPPA)
    h.estimate()
    return h


def switch(h, mode):
    for op in h.levels:
        op.set_tensor_cores(mode)


def cycle(h, b):
    x = torch.empty_like(b)
    h.mg.vmult(x, b)
    return x


def distance(a, b):
    return float((a - b).norm() / b.norm())


def test_switch_between_cycles():
    h = hierarchy()
    b = h.levels[-1].assemble_rhs(0)
    b = b * (1.0 + 0.5 * torch.rand_like(b))
    plain = cycle(h, b)
    other = hierarchy()
    switch(other, 1)
    effect = distance(cycle(other, b), plain)
    assert effect > 1e-4
    for _ in range(2):
        switch(h, 0)
        for _ in range(2):
            assert distance(cycle(h, b), plain) < 1e-5
        switch(h, 1)
        for _ in range(2):
            assert 0.5 * effect < distance(cycle(h, b), plain) < 2.0 * effect
