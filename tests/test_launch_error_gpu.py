"""GPU test of the error state after a failed launch: a solve on the legacy default
stream is refused by the runtime while a blocking stream captures; the call
returns FF_ERR_CUDA, and calls after it are as if it had not been made."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

RELAXED = 2   # cudaStreamCaptureModeRelaxed


@pytest.mark.parametrize("n", [(64, 64, 64), (30, 45, 50), (32, 32, 41)])
def test_calls_after_a_refused_launch(torch_cuda, ff, n):
    torch = torch_cuda
    plan = ff.Plan(n)
    size, N = plan.nbytes // 8, n[0] * n[1] * n[2]
    f = torch.randn(N, dtype=torch.float64, device="cuda")
    d, p = (torch.zeros(size, dtype=torch.float64, device="cuda") for _ in range(2))
    d[:N] = f
    plan.solve(d, p)
    want = p[:N].clone()
    d[:N] = f
    torch.cuda.synchronize()

    rt = ctypes.CDLL("libcudart.so.12")
    s, g = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(s)) == 0
    assert rt.cudaStreamBeginCapture(s, RELAXED) == 0
    try:
        with pytest.raises(ff.FFError) as e:
            plan.solve(d, p)
        left = rt.cudaPeekAtLastError()
    finally:
        rt.cudaStreamEndCapture(s, ctypes.byref(g))   # the refused launch has invalidated it
        rt.cudaStreamDestroy(s)
        rt.cudaGetLastError()
    assert e.value.status == ff.FF_ERR_CUDA
    assert left == 0   # the next launch's check does not report it again

    again = ff.Plan(n)
    again.solve(d, p)
    torch.cuda.synchronize()
    assert torch.equal(p[:N], want)
    batch = ff.Batch([(8, 8, 8)])
    x, y = (torch.zeros(batch.nbytes[0] // 8, dtype=torch.float64, device="cuda") for _ in range(2))
    batch.solve([x], [y])
