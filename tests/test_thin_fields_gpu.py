"""GPU tests of the field kernels on grids whose tiles (64 lines by at most 64
points along z) would be mostly empty: both sides of the rule that sends them
point by point, against the same formulas in numpy, and the time of a single line
or of one point along z against that of a cube of as many points."""
import pytest

from test_field_gpu import test_fields_and_sums_match_the_formulas as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("modes", [0, 3, 64])
@pytest.mark.parametrize("n", [(9, 8, 1), (40, 30, 3), (40, 30, 4), (13, 11, 5), (13, 11, 6), (13, 11, 7), (13, 11, 8),
                               (1, 1, 64), (1, 3, 500), (2, 2, 500), (5, 1, 320), (1, 7, 320), (2, 4, 320), (3, 3, 320),
                               (2, 5, 320), (1, 11, 320)])
def test_both_sides_of_the_rule(torch_cuda, ff, n, modes, precision):
    check(torch_cuda, ff, n, modes, precision)


@pytest.mark.parametrize("modes", [0, 64])
@pytest.mark.parametrize("n", [(1, 1, 144 ** 3), (1728, 1728, 1)])
def test_thin_grids_take_the_time_of_their_points(torch_cuda, ff, n, modes):
    torch = torch_cuda
    md = [(1 + q % 5, q % 3, q % 7, 0.1, 0.2) for q in range(modes)]

    def time(n):
        f = torch.empty(n, dtype=torch.float64, device="cuda")
        best = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                ff.init_field(n, f, md)
                ff.error_sums(n, f, md)
            b.record()
            b.synchronize()
            best.append(a.elapsed_time(b))
        return min(best)

    # a point of its own costs a cosine per mode and nine transcendentals, about
    # seven times a tile's point; in tiles these grids took 40 times as long
    assert time(n) <= 15.0 * time((144, 144, 144))
