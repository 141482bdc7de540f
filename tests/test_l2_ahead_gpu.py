"""GPU tests of FF_L2_AHEAD (the z passes' L2 prefetch distance in blocks, read at
plan creation): compile-time and generic lengths take it alike, and results do
not depend on it."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def l2_ahead(ff, plan):
    # internal to the library: ff::plan_l2_ahead(const ff_plan *)
    fn = ff.lib()._ZN2ff13plan_l2_aheadEPK7ff_plan
    fn.argtypes, fn.restype = [ctypes.c_void_p], ctypes.c_int
    return fn(plan._h)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(48, 40, 64), (48, 40, 60), (48, 40, 27), (160, 160, 6)])
def test_distance_of_every_kind_of_z_pass(torch_cuda, ff, monkeypatch, n, precision):
    torch = torch_cuda
    dt = torch.float64 if precision == 0 else torch.float32
    f = torch.randn(n[0] * n[1] * n[2], dtype=dt, device="cuda")
    results = []
    for value in (None, "0", "1", "37", "100000"):
        if value is None:
            monkeypatch.delenv("FF_L2_AHEAD", raising=False)
        else:
            monkeypatch.setenv("FF_L2_AHEAD", value)
        plan = ff.Plan(n, precision=precision)
        if value is None:
            assert l2_ahead(ff, plan) > 0
        else:
            assert l2_ahead(ff, plan) == int(value)
        d, p = (torch.zeros(plan.nbytes // f.element_size(), dtype=dt, device="cuda") for _ in range(2))
        d[:f.numel()] = f
        plan.solve(d, p)
        results.append(p[:f.numel()].clone())
    for r in results[1:]:
        assert torch.equal(r, results[0])
