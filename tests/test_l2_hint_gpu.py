"""GPU tests of the z passes' L2 hints (the input of the tile one resident wave
ahead) where that tile is a last one of a single line of fewer than 16 bytes:
225 x 257 lines are one more than a multiple of every tile's lines and more
than a wave of them.  Against numpy's FFTs of the same input.

FP64 bar: 1e-12 relative L2; FP32: 1e-5."""
import pytest

from test_gen_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nk", [1, 2, 3, 4, 5])
def test_last_tile_of_one_short_line(torch_cuda, ff, nk, precision):
    check(torch_cuda, ff, (225, 257, nk), precision)
