"""GPU tests of the field kernels' tiles (64 lines by at most 64 points along
z, whose factors and mode phases come from tables): the right-hand side and
the error sums at the edges of lines, chunks and mode counts, against the same
formulas (FishFry.hpp:22-44, :71-101) point by point in numpy."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def point_by_point(n, modes):
    x, y, z = (-math.pi + np.arange(m) * (2.0 * math.pi / m) for m in n)
    cx, sx, cy, sy, cz, sz = np.cos(x), np.sin(x), np.cos(y), np.sin(y), np.cos(z), np.sin(z)
    px, py, pz = cx * np.exp(sx), sy * np.exp(cy), cz * np.exp(cz)
    dx = -np.exp(sx) * sx * cx * (sx + 3.0)
    dy = sy * np.exp(cy) * (sy * sy - 3.0 * cy - 1.0)
    dz = np.exp(cz) * (3.0 * sz * sz - cz * cz * cz - 1.0)

    def ax(a, b, c):
        return a[:, None, None] * b[None, :, None] * c[None, None, :]

    f = ax(px, py, dz) + ax(px, dy, pz) + ax(dx, py, pz)
    phi = ax(px, py, pz)
    for kx, ky, kz, a, theta in modes:
        k2 = kx * kx + ky * ky + kz * kz
        if k2 == 0:
            continue
        c = np.cos(kx * x[:, None, None] + ky * y[None, :, None] + kz * z[None, None, :] + theta)
        f += a * c
        phi -= a / k2 * c
    return f, phi


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("modes", [0, 3, 64])
@pytest.mark.parametrize("n", [(1, 1, 1), (2, 3, 5), (8, 8, 64), (5, 13, 63), (9, 7, 65), (3, 22, 128), (4, 33, 129),
                               (1, 1, 75841)])
def test_fields_and_sums_match_the_formulas(torch_cuda, ff, n, modes, precision):
    torch = torch_cuda
    rng = np.random.default_rng(n[2] + modes)
    md = [(int(a), int(b), int(c), float(w), float(t)) for a, b, c, w, t in
          zip(*rng.integers(-32, 33, (3, modes)), rng.normal(0, 0.1, modes), rng.uniform(0, 2 * math.pi, modes))]
    if modes:
        md[0] = (0, 0, 0, 1.0, 0.5)   # counts as absent
    f, phi = point_by_point(n, md)
    # the phase of a mode is at most 3 * 32 * pi + 2 * pi < 320, rounded a few
    # times on each side; the analytic sums are below 100 in magnitude
    tol = 64 * EPS * (100.0 + 320.0 * sum(abs(m[3]) for m in md))
    dt = torch.float64 if precision == 0 else torch.float32
    got = torch.empty(n, dtype=dt, device="cuda")
    ff.init_field(n, got, md, precision)
    d = np.abs(got.double().cpu().numpy() - f).max()
    assert d <= tol + (2.0 ** -23 * np.abs(f).max() if precision else 0.0)
    p = torch.from_numpy(phi + rng.normal(0, 0.1, n)).cuda().to(dt)
    e = np.abs(phi - p.double().cpu().numpy())
    sums = ff.error_sums(n, p, md, precision)
    assert abs(sums[0] - e.sum()) <= e.size * tol
    assert abs(sums[1] - (e * e).sum()) <= 2 * e.size * tol * (e.max() + tol)
    assert abs(sums[2] - e.max()) <= tol
    assert sums == ff.error_sums(n, p, md, precision)     # a fixed order: the same sums again
    p.view(-1)[-1] = float("nan")
    assert math.isnan(ff.error_sums(n, p, md, precision)[2])
