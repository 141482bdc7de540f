"""GPU tests of a server's descriptor slots: a new server does not hold max_active of
them, and requests beyond the first slots (256, 512, ... per precision) are served
like the others, while earlier ones are in flight."""
import pytest

pytestmark = pytest.mark.gpu


def test_a_new_server_holds_few_slots(torch_cuda, ff):
    torch = torch_cuda
    ff.Server(1 << 20, max_active=4).close()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    srv = ff.Server(1 << 20, max_active=65536)
    used = free0 - torch.cuda.mem_get_info()[0]
    srv.close()
    # the work lists of three steps and five passes for 65536 members: 12 bytes a
    # member, twice (precisions); the budget; pages of 2 MB
    assert used <= 2 * 3 * 5 * 65536 * 12 + (1 << 20) + (12 << 20), used


@pytest.mark.parametrize("count,max_active", [(257, 4096), (700, 4096), (700, 300), (700, 1), (1100, 1024)])
def test_requests_beyond_the_first_slots(torch_cuda, ff, count, max_active):
    torch = torch_cuda
    dims = [(8, 9, 10), (16, 6, 5), (4, 4, 32), (7, 3, 12)]
    plans = {(n, p): ff.Plan(n, precision=p) for n in dims for p in (0, 1)}
    reqs = []
    for q in range(count):
        n, p = dims[q % 4], (q // 4) % 2
        dt = torch.float64 if p == 0 else torch.float32
        reqs.append((n, p, torch.randn(n, dtype=dt, device="cuda", generator=torch.Generator("cuda").manual_seed(q))))
    torch.cuda.synchronize()
    srv = ff.Server(1 << 28, max_active=max_active)
    try:
        # results stay in their slots until they are fetched: all of them are taken
        # at once where max_active allows it
        ids = [srv.submit(n, f, p) for n, p, f in reqs]
        out = [torch.empty_like(f) for _, _, f in reqs]
        at = {i: q for q, i in enumerate(ids)}
        if max_active >= count:
            for i in ids:
                srv.wait(i, 60_000.0)
        for _ in range(count):
            i = srv.next(60_000.0)[0]
            srv.fetch(i, out[at[i]])
        srv.check()
    finally:
        srv.close()
    for (n, p, f), phi in zip(reqs, out):
        plan = plans[(n, p)]
        d, r = (torch.zeros(plan.nbytes // f.element_size(), dtype=f.dtype, device="cuda") for _ in range(2))
        d[:f.numel()] = f.reshape(-1)
        plan.solve(d, r)
        w = r[:f.numel()].view(n)
        e = float((phi.double() - w.double()).norm() / w.double().norm())
        assert e <= (1e-12 if p == 0 else 1e-5), (n, p, e)
