"""A call that CUDA refuses raises its error once: the calls after it run."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
import pmg  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm", [True, False])
def test_reduction_on_a_stream_being_captured(warm):
    rt = ctypes.CDLL("libcudart.so.12")
    op = pmg.LaplaceOperator(pmg.Mesh(pmg.Box.make(refine=2)), 2, pmg.F64)
    x = torch.ones(op.m(), device="cuda", dtype=torch.float64)
    if warm:
        pmg.vector_dot(x, x)
    side, graph = torch.cuda.Stream(), ctypes.c_void_p()
    torch.cuda.synchronize()
    handle = ctypes.c_void_p(side.cuda_stream)
    for _ in range(6):  # more often than there is reduction memory kept for reuse
        assert rt.cudaStreamBeginCapture(handle, 1) == 0  # thread-local mode
        with torch.cuda.stream(side):
            with pytest.raises(pmg.PmgError):
                pmg.vector_dot(x, x)
        assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) != 0
        rt.cudaGetLastError()
        op.compute_diagonal()  # (its launches are followed by a look at CUDA's last error)
        assert pmg.vector_dot(x, x) == op.m()
    with torch.cuda.stream(side):
        assert pmg.vector_dot(x, x) == op.m()
