"""GPU tests of Fourier modes that are not ordinary numbers in the right-hand side
and the error sums: infinite and NaN amplitudes, and a zero mode (which counts
as absent) with a phase or amplitude that is not finite.  Against the formula
point by point in numpy."""
import math

import numpy as np
import pytest

from test_field_gpu import point_by_point

pytestmark = pytest.mark.gpu

INF, NAN = math.inf, math.nan


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("modes", [
    [(1, 2, 3, INF, 0.7)],
    [(0, 0, 1, -INF, 0.3), (2, 0, 0, 0.5, 0.1)],
    [(1, 0, 0, 0.25, 0.2), (0, 3, 1, NAN, 0.2)],
    [(0, 0, 0, 1.0, NAN), (1, 2, 0, 0.5, 0.25)],
    [(0, 0, 0, INF, INF), (1, 2, 0, 0.5, 0.25)],
])
def test_modes_that_are_not_finite(torch_cuda, ff, modes, precision):
    torch, n = torch_cuda, (5, 9, 66)
    with np.errstate(all="ignore"):
        f, phi = point_by_point(n, modes)
    # points whose infinite mode's cosine is not within rounding of zero
    clear = np.ones(n, dtype=bool)
    x, y, z = (-math.pi + np.arange(m) * (2.0 * math.pi / m) for m in n)
    for kx, ky, kz, a, theta in modes:
        if math.isinf(a) and (kx, ky, kz) != (0, 0, 0):
            c = np.cos(kx * x[:, None, None] + ky * y[None, :, None] + kz * z[None, None, :] + theta)
            clear &= np.abs(c) > 1e-9
    assert clear.sum() > 0.9 * clear.size
    dt = torch.float64 if precision == 0 else torch.float32
    got = torch.empty(n, dtype=dt, device="cuda")
    ff.init_field(n, got, modes, precision)
    got = got.double().cpu().numpy()
    # finite points: sums of terms below 100, as the analytic field's
    tol = 1e-12 if precision == 0 else 2.0 ** -23 * 100.0
    assert np.allclose(got[clear], f[clear], rtol=0.0, atol=tol, equal_nan=True)
    with np.errstate(all="ignore"):
        want = [np.abs(phi).sum(), (phi * phi).sum(), np.abs(phi).max()]
    sums = ff.error_sums(n, None, modes, precision)
    assert np.allclose(sums, want, rtol=1e-12, atol=0.0, equal_nan=True), (sums, want)
