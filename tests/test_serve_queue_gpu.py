"""GPU test of a server's queue when it grows past the admission window (64
requests): everything submitted is served although no result is fetched before the
last one is done.  Matrix products that fill the GPU keep the scheduler in its
first admission pass, where it waits for the tables of the first request's axes,
while the others are submitted."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_a_queue_longer_than_the_admission_window(torch_cuda, ff, precision):
    torch = torch_cuda
    dt = torch.float64 if precision == 0 else torch.float32
    dims = [(4, 4, 8)] * 300
    fields = [torch.randn(n, dtype=dt, device="cuda") for n in dims]
    a = torch.randn((8192, 8192), dtype=torch.float64, device="cuda")
    b = torch.mm(a, a)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    srv = ff.Server(1 << 30, max_active=1024)
    try:
        with torch.cuda.stream(side):
            for _ in range(4):
                torch.mm(a, a, out=b)
        ids = [srv.submit(n, f, precision) for n, f in zip(dims, fields)]
        for i in ids:
            srv.wait(i, 20_000.0)
        out = torch.empty((4, 4, 8), dtype=dt, device="cuda")
        srv.fetch(ids[-1], out)
        srv.check()
    finally:
        srv.close()
    plan = ff.Plan((4, 4, 8), precision=precision)
    d, p = (torch.zeros(plan.nbytes // out.element_size(), dtype=dt, device="cuda") for _ in range(2))
    d[:128] = fields[-1].reshape(-1)
    plan.solve(d, p)
    want = p[:128].view(4, 4, 8)
    assert float((out - want).norm() / want.norm()) <= (1e-12 if precision == 0 else 1e-5)
