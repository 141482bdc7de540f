"""GPU tests of the passes along axes without a compile-time plan (ff_gen_dev.cuh)
at the lengths where their plans and tiles change: every radix first, last and
alone, one to five stages, odd lengths (lines moved as one block), partly
filled units and tiles, 128-, 64- and 32-byte rows, TMA boxes that reach past
the line.  Against numpy's FFTs of the same input.

FP64 bar: 1e-12 relative L2; FP32: 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHORT = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 35, 36, 40, 42, 45, 48, 49,
         50, 54, 56, 60, 63, 70, 72, 80, 81, 84, 90, 96, 98, 100, 105, 108, 120, 125, 126, 135, 140, 144, 147, 150, 160,
         162, 168, 175, 180, 189, 192, 196, 200, 210, 216, 224, 225, 240, 243, 245, 250, 252, 270, 280, 288, 294, 300,
         320, 324, 336, 343, 350, 360, 375, 378, 384, 392, 400, 405, 420, 432, 441, 448, 450, 480, 486, 490, 500, 504,
         525, 540, 560, 567, 576, 588, 600, 625, 630, 640, 686, 700, 720, 729, 750, 768, 800]
LONG = [810, 900, 960, 1000, 1080, 1125, 1200, 1225, 1280, 1344, 1500, 1536, 1715, 1800, 1920, 2000, 2025, 2048, 2187,
        2401, 2500, 3000, 3125, 3375, 3500, 3600, 3645, 3888, 3969, 4000, 4050, 4096]


def solve_numpy(f, dd):
    s = np.fft.rfftn(f)
    ni, nj, nk = f.shape
    i, j, k = np.arange(ni), np.arange(nj), np.arange(nk // 2 + 1)
    k2 = (((np.minimum(i, ni - i) * dd[0]) ** 2)[:, None, None] + ((np.minimum(j, nj - j) * dd[1]) ** 2)[None, :, None]
          + ((k * dd[2]) ** 2)[None, None, :])
    k2[0, 0, 0] = 1.0
    s /= -k2
    s[0, 0, 0] = 0.0
    return np.fft.irfftn(s, s=f.shape, axes=(0, 1, 2))


def check(torch, ff, n, precision):
    rng = np.random.default_rng(n[0] * 31 + n[1] * 7 + n[2] + precision)
    f = rng.standard_normal(n)
    f -= f.mean()
    if precision:
        f = f.astype(np.float32).astype(np.float64)
    lo = [-1.0, 0.5, 2.0]
    hi = [lo[a] + (1.0 + a) * max(n[a] - 1, 1) / n[a] for a in range(3)]
    dd = [2 * np.pi * (n[a] - 1) / (n[a] * (hi[a] - lo[a])) if n[a] > 1 else 0.0 for a in range(3)]
    plan = ff.Plan(n, lo, hi, precision)
    dt = torch.float64 if precision == 0 else torch.float32
    size = plan.nbytes // (8 if precision == 0 else 4)
    # guard zones: nothing outside the caller's buffers is written
    guard = 4096
    d = torch.full((size + 2 * guard,), 7.5, dtype=dt, device="cuda")
    p = torch.full((size + 2 * guard,), 7.5, dtype=dt, device="cuda")
    N = f.size
    d[guard:guard + N] = torch.from_numpy(f.ravel()).cuda().to(dt)
    plan.solve(d[guard:guard + size], p[guard:guard + size])
    plan.check()
    for b in (d, p):
        assert bool((b[:guard] == 7.5).all()) and bool((b[guard + size:] == 7.5).all())
    got = p[guard:guard + N].double().cpu().numpy().reshape(n)
    want = solve_numpy(f, dd)
    err = np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-300)
    assert err <= (1e-12 if precision == 0 else 1e-5) or N == 1, err


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_every_short_length(torch_cuda, ff, axis, precision):
    for q, m in enumerate(SHORT):
        a, b = [(6, 10), (5, 27), (9, 33), (4, 21)][q % 4]
        n = {0: (m, a, b), 1: (a, m, b), 2: (a, b, m)}[axis]
        check(torch_cuda, ff, n, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_long_lengths(torch_cuda, ff, axis, precision):
    for q, m in enumerate(LONG):
        a, b = [(3, 10), (2, 7)][q % 2]
        n = {0: (m, a, b), 1: (a, m, b), 2: (a, b, m)}[axis]
        check(torch_cuda, ff, n, precision)


# Bluestein axes: the smallest, odd and even, just below and above a change of
# the tile's row width, the largest of the declared range
FACTORS = [11, 13, 17, 22, 26, 31, 33, 34, 37, 44, 55, 61, 66, 77, 88, 97, 101, 110, 121, 127, 130, 143, 169, 187, 211,
           241, 251, 254, 257, 289, 290, 293, 296, 307, 331, 341, 374, 419, 499, 509, 601, 701, 883, 887, 901]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_lengths_with_larger_prime_factors(torch_cuda, ff, axis, precision):
    for q, m in enumerate(FACTORS):
        a, b = [(6, 10), (5, 27), (9, 33), (4, 21)][q % 4]
        n = {0: (m, a, b), 1: (a, m, b), 2: (a, b, m)}[axis]
        check(torch_cuda, ff, n, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(100, 90, 81), (96, 75, 80), (147, 98, 105), (200, 180, 160)])
def test_grids_of_several_waves(torch_cuda, ff, n, precision):
    check(torch_cuda, ff, n, precision)


# Passes launched as programmatic dependents of one another: results of solves
# queued back to back on shared buffers, on the default and a side stream, and
# replayed from a captured graph.
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(64, 64, 64), (30, 45, 50), (33, 34, 35)])
def test_chained_passes_back_to_back_and_captured(torch_cuda, ff, n, precision):
    torch = torch_cuda
    dt = torch.float64 if precision == 0 else torch.float32
    plan = ff.Plan(n, precision=precision)
    size, N = plan.nbytes // (8 if precision == 0 else 4), n[0] * n[1] * n[2]
    fields = [torch.randn(N, dtype=dt, device="cuda") for _ in range(4)]
    d, p = (torch.zeros(size, dtype=dt, device="cuda") for _ in range(2))
    want = []
    for f in fields:
        d[:N] = f
        torch.cuda.synchronize()
        plan.solve(d, p)
        torch.cuda.synchronize()
        want.append(p[:N].clone())

    def run(stream):
        out = []
        for f in fields:
            d[:N].copy_(f)
            plan.solve(d, p, stream=stream)
            out.append(p[:N].clone())
        return out

    side = torch.cuda.Stream()
    got = run(None)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got += run(side)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run(torch.cuda.current_stream())
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for q, out in enumerate(got + captured):
        assert torch.equal(out, want[q % len(fields)]), q
