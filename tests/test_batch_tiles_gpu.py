"""GPU tests of the batch tiles of runtime plans and of FP32 column pairs: every
radix first and last, one to six stages, odd lengths (lines moved by the threads,
padded spectrum rows), odd numbers of FP32 line pairs per tile, more grids than
one step of the entry search covers.  Against the single-grid plan of each grid,
which runs other kernels (FP64 within 1e-13 relative L2, FP32 within 2e-6: both
sides round each transform of at most 574 points a few dozen times), under the
default and the tuned shapes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 35, 36, 40, 42, 45, 48, 49,
           50, 54, 56, 60, 63, 64, 70, 72, 75, 80, 81, 84, 90, 96, 98, 100, 105, 108, 112, 120, 125, 126, 128, 135, 140,
           144, 147, 150, 160, 162, 189, 200, 210, 243, 250, 256, 270, 288, 300, 320, 343, 375, 400, 441, 486, 500, 512,
           567]


def dims_with(axis):
    others = [(6, 10), (5, 27), (9, 33), (4, 21), (12, 15)]
    out = []
    for q, m in enumerate(LENGTHS):
        a, b = others[q % len(others)]
        out.append({0: (m, a, b), 1: (a, m, b), 2: (a, b, m)}[axis])
    return out


def solve_and_compare(torch, ff, dims, precision, tuned=False):
    dt = torch.float64 if precision == 0 else torch.float32
    esz = 8 if precision == 0 else 4
    batch = ff.Batch(dims, precision=precision)
    d = [torch.zeros(b // esz, dtype=dt, device="cuda") for b in batch.nbytes]
    p = [torch.zeros_like(x) for x in d]
    if tuned:
        batch.tune(d, p, reps=1)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(len(dims) + precision)
    fs = [torch.randn(n[0] * n[1] * n[2], dtype=dt, device="cuda", generator=gen) for n in dims]
    for x, f in zip(d, fs):
        x[:f.numel()] = f
    batch.solve(d, p)
    batch.check()
    for g, n in enumerate(dims):
        plan = ff.Plan(n, precision=precision)
        dd = torch.zeros_like(d[g])
        dd[:fs[g].numel()] = fs[g]
        pp = torch.zeros_like(dd)
        plan.solve(dd, pp)
        a = p[g][:fs[g].numel()].double().cpu().numpy()
        b = pp[:fs[g].numel()].double().cpu().numpy()
        err = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)
        assert err <= (1e-13 if precision == 0 else 2e-6), (n, err)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_every_length(torch_cuda, ff, axis, precision):
    solve_and_compare(torch_cuda, ff, dims_with(axis), precision)


@pytest.mark.parametrize("precision", [0, 1])
def test_tuned_shapes(torch_cuda, ff, precision):
    solve_and_compare(torch_cuda, ff, [(64, 64, 64), (96, 48, 80), (32, 128, 54), (25, 45, 49), (100, 72, 56)], precision,
                      tuned=True)


@pytest.mark.parametrize("precision", [0, 1])
def test_more_grids_than_a_search_step(torch_cuda, ff, precision):
    rng = np.random.default_rng(3)
    choices = [1, 3, 4, 7, 8, 12, 15, 16, 32]
    solve_and_compare(torch_cuda, ff, [tuple(int(x) for x in rng.choice(choices, 3)) for _ in range(75)], precision)
