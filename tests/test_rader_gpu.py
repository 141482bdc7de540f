"""GPU tests of axes of a prime length n whose n - 1 has only the factors 2, 3, 5
and 7: a convolution of n - 1 points instead of Bluestein's (ff_bluestein.hpp).
Every such length up to 500 and long ones, on each axis, the last lengths before and
after the rule's lower end, several such axes at once.  Against numpy's FFTs of
the same input (test_gen_gpu.check).

FP64 bar: 1e-12 relative L2; FP32: 1e-5."""
import pytest

from test_gen_gpu import check

pytestmark = pytest.mark.gpu


def smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


PRIMES = [n for n in range(11, 500) if all(n % q for q in range(2, n)) and smooth(n - 1)]
LONG = [641, 757, 1009, 1373, 1601, 2017, 2593, 3001]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_prime_lengths(torch_cuda, ff, axis, precision):
    for q, m in enumerate(PRIMES):
        a, b = [(6, 10), (5, 27), (9, 33), (4, 21)][q % 4]
        check(torch_cuda, ff, {0: (m, a, b), 1: (a, m, b), 2: (a, b, m)}[axis], precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_long_prime_lengths(torch_cuda, ff, axis, precision):
    for q, m in enumerate(LONG):
        a, b = [(3, 10), (2, 7)][q % 2]
        check(torch_cuda, ff, {0: (m, a, b), 1: (a, m, b), 2: (a, b, m)}[axis], precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(13, 11, 17), (127, 113, 109), (97, 64, 211), (61, 59, 73)])
def test_several_prime_axes(torch_cuda, ff, n, precision):
    check(torch_cuda, ff, n, precision)


# 3889 = 2^4 3^5 + 1 points: Bluestein's tile does not fit, so the length is refused
@pytest.mark.parametrize("n", [(3889, 4, 4), (4, 3889, 4)])
def test_lengths_beyond_bluestein_stay_refused(torch_cuda, ff, n):
    with pytest.raises(ff.FFError) as e:
        ff.Plan(n)
    assert e.value.status == ff.FF_ERR_UNSUPPORTED
