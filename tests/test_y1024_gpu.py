"""GPU tests of the FP32 y passes of 1024 points (stages 16 x 8 x 8, ff_fft.cuh):
few and many planes, one partly filled tile, an odd column left over, several tiles.
Against numpy's FFTs of the same input (test_gen_gpu.check).  FP32 bar: 1e-5
relative L2."""
import pytest

from test_gen_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1024, 2), (3, 1024, 14), (2, 1024, 16), (5, 1024, 33), (64, 1024, 64), (9, 1024, 251),
                               (1024, 1024, 8)])
def test_fp32_y_of_1024_points(torch_cuda, ff, n):
    check(torch_cuda, ff, n, 1)
