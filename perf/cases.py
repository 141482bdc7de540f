"""What the framework's speed is measured on: calls a user's program makes,
through the public entry points, over the sizes and options it takes.

A case is a dict of plain values; `kind` says which call it is:

  solve    Plan.solve of one grid: the field f of a time step is put into the
           density buffer (a solve overwrites it), the solve is enqueued, phi
           is read from the potential buffer
  plugin   the same through ParisPencil, the reference's plugin interface,
           which blocks until phi is there and returns its time stamps
  batch    Batch.solve of many grids of uneven sizes
  serve    a burst of requests of mixed sizes and precisions to a Server
  fields   the harness's own device work: the analytic right-hand side (with
           seeded Fourier modes or without) and the error norms of a given phi
"""
import math
import random

import torch

import fishfry_b200 as ff

FP64, FP32 = ff.FF_FP64, ff.FF_FP32
DEV = "cuda"


def _dtype(precision):
    return torch.float64 if precision == "fp64" else torch.float32


def _code(precision):
    return FP64 if precision == "fp64" else FP32


def listed():
    return [
        # a small solver call inside a host program: launches and latency
        dict(name="plugin_32cube_fp64", kind="plugin", ni=32, nj=32, nk=32, precision="fp64"),
        # a small production grid, power of two
        dict(name="solve_128cube_fp64", kind="solve", ni=128, nj=128, nk=128, precision="fp64"),
        # a small grid of mixed 5-smooth lengths, as serving mixes and user meshes have
        dict(name="solve_200x180x160_fp32", kind="solve", ni=200, nj=180, nk=160, precision="fp32"),
        # a ragged grid: one prime axis, the others powers of two
        dict(name="solve_256x256x251_fp64", kind="solve", ni=256, nj=256, nk=251, precision="fp64"),
        # a large grid of 5-smooth lengths that are not powers of two
        dict(name="solve_480x400x360_fp64", kind="solve", ni=480, nj=400, nk=360, precision="fp64"),
        # the benchmark's grid, and the same in FP32
        dict(name="solve_512cube_fp64", kind="solve", ni=512, nj=512, nk=512, precision="fp64"),
        dict(name="solve_512cube_fp32", kind="solve", ni=512, nj=512, nk=512, precision="fp32"),
        # the largest grid of the benchmark
        dict(name="solve_1024cube_fp32", kind="solve", ni=1024, nj=1024, nk=1024, precision="fp32"),
        # many small grids at once: the benchmark's batch mix, fewer grids
        dict(name="batch_mix_fp32", kind="batch", grids=60, lengths="32,48,64,80,96,128", dims_seed=2024,
             precision="fp32"),
        # many small grids of arbitrary smooth lengths, odd ones and a factor of 7 among them
        dict(name="batch_ragged_fp64", kind="batch", grids=48, lengths="24,30,45,56,72,100,108,125,144,160",
             dims_seed=7, precision="fp64"),
        # a burst of service requests, FP32 and FP64 in turn
        dict(name="serve_burst", kind="serve", requests=40, max_axis=256, max_points=1 << 22, dims_seed=12345),
        # the harness around a solve: right-hand side and error norms
        dict(name="fields_256cube_fp64", kind="fields", ni=256, nj=256, nk=256, precision="fp64", modes=0),
    ]


# ------------------------------------------------------------------ sizes
def _smooth(n, primes=(2, 3, 5, 7)):
    for p in primes:
        while n % p == 0:
            n //= p
    return n == 1


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axis(rng, lo, hi, style):
    """A length in [lo, hi], even over its logarithm: any, 2^a 3^b 5^c 7^d, or a power of two."""
    for _ in range(1000):
        n = max(lo, min(hi, _log_int(rng, lo, hi)))
        if style == "pow2":
            return 1 << max(int(math.ceil(math.log2(lo))), min(int(math.log2(hi)), int(round(math.log2(n)))))
        if style == "any" or _smooth(n):
            return n
    return lo


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["plugin", "batch", "serve", "fields"])
    precision = rng.choice(["fp64", "fp32"])
    if kind in ("solve", "plugin"):
        style = rng.choice(["smooth", "smooth", "pow2", "any"])
        hi, most = {"pow2": (1024, 1 << 28), "smooth": (768, 1 << 27), "any": (420, 1 << 24)}[style]
        if kind == "plugin":
            hi, most = min(hi, 128), 1 << 21
        while True:
            n = [_axis(rng, 16, hi, style) for _ in range(3)]
            if n[0] * n[1] * n[2] <= most:
                break
        return dict(kind=kind, ni=n[0], nj=n[1], nk=n[2], precision="fp64" if kind == "plugin" else precision)
    if kind == "batch":
        lengths = sorted({_axis(rng, 24, 160, "smooth") for _ in range(8)})
        return dict(kind=kind, grids=rng.randint(12, 60), lengths=",".join(map(str, lengths)),
                    dims_seed=rng.randrange(1 << 20), precision=precision)
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(8, 48), max_axis=rng.choice([96, 160, 256]), max_points=1 << 22,
                    dims_seed=rng.randrange(1 << 20))
    n = [_axis(rng, 24, 320, "any") for _ in range(3)]
    return dict(kind=kind, ni=n[0], nj=n[1], nk=n[2], precision=precision, modes=rng.choice([0, 0, 8, 64]))


def _dims_of(case):
    """Grids of a batch or serve case: (ni, nj, nk, precision) each."""
    r = random.Random(case["dims_seed"])
    if case["kind"] == "batch":
        choices = [int(x) for x in case["lengths"].split(",")]
        return [tuple(r.choice(choices) for _ in range(3)) + (case["precision"],) for _ in range(case["grids"])]
    got = []
    while len(got) < case["requests"]:
        n = tuple(_axis(r, 32, case["max_axis"], "smooth") for _ in range(3))
        if n[0] * n[1] * n[2] <= case["max_points"]:
            got.append(n + ("fp32" if len(got) % 2 else "fp64",))
    return got


# ----------------------------------------------------------------- inputs
def _field(gen, count, dtype):
    """A right-hand side: a density contrast with power at every wavenumber."""
    return torch.randn(count, generator=gen, device=DEV, dtype=dtype)


def _modes(case, seed):
    """Seeded Fourier modes (kx, ky, kz, a, theta), below every axis's Nyquist wavenumber."""
    r = random.Random(seed)
    top = [min(32, (case[a] - 1) // 2) for a in ("ni", "nj", "nk")]
    got = []
    while len(got) < case["modes"]:
        k = [r.randint(-t, t) for t in top]
        if any(k):
            got.append((k[0], k[1], k[2], r.gauss(0.0, 0.1), r.uniform(0.0, 2 * math.pi)))
    return got


def _analytic(n, modes, solution):
    """The harness's f or phi on its grid (FishFry.hpp:22-44, :71-86), plus the modes', in FP64."""
    x, y, z = (-math.pi + torch.arange(m, device=DEV, dtype=torch.float64) * (2.0 * math.pi / m) for m in n)
    cx, sx, cy, sy, cz, sz = x.cos(), x.sin(), y.cos(), y.sin(), z.cos(), z.sin()
    px, py, pz = cx * sx.exp(), sy * cy.exp(), cz * cz.exp()
    dx = -sx.exp() * sx * cx * (sx + 3.0)
    dy = sy * cy.exp() * (sy * sy - 3.0 * cy - 1.0)
    dz = cz.exp() * (3.0 * sz * sz - cz * cz * cz - 1.0)
    ax = lambda u, v, w: u[:, None, None] * v[None, :, None] * w[None, None, :]  # noqa: E731
    got = ax(px, py, pz) if solution else ax(px, py, dz) + ax(px, dy, pz) + ax(dx, py, pz)
    for kx, ky, kz, a, theta in modes:
        w = -a / (kx * kx + ky * ky + kz * kz) if solution else a
        got += w * torch.cos((kx * x + theta)[:, None, None] + (ky * y)[None, :, None] + (kz * z)[None, None, :])
    return got


def _inputs(case, seed):
    """Inputs alone (what `exact` needs too): the fields, or modes and phi."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    if case["kind"] in ("solve", "plugin"):
        return _field(gen, case["ni"] * case["nj"] * case["nk"], _dtype(case["precision"]))
    if case["kind"] in ("batch", "serve"):
        return [_field(gen, d[0] * d[1] * d[2], _dtype(d[3])) for d in _dims_of(case)]
    n = (case["ni"], case["nj"], case["nk"])
    modes = _modes(case, seed)
    phi = _analytic(n, modes, True).reshape(-1)
    phi += 1e-3 * torch.randn(phi.numel(), generator=gen, device=DEV, dtype=torch.float64)
    return modes, phi.to(_dtype(case["precision"]))


def prepare(case, seed):
    kind = case["kind"]
    state = dict(kind=kind)
    if kind in ("solve", "plugin"):
        n = (case["ni"], case["nj"], case["nk"])
        f = _inputs(case, seed)
        if kind == "plugin":
            lo, hi, _, _ = ff.reference_domain(n)
            plan = ff.ParisPencil(n, lo, hi)
        else:
            plan = ff.Plan(n, precision=_code(case["precision"]))
        size = plan.bytes() // f.element_size()
        density, potential = (torch.empty(size, device=DEV, dtype=f.dtype) for _ in range(2))
        state.update(plan=plan, f=f, whole=potential, potential=potential[:f.numel()].view(n), density=density,
                     into=density[:f.numel()])
    elif kind == "batch":
        dims = [d[:3] for d in _dims_of(case)]
        batch = ff.Batch(dims, precision=_code(case["precision"]))
        fields = _inputs(case, seed)
        each = fields[0].element_size()
        # every grid's buffers in one allocation (16-byte aligned starts), so
        # that a step's fields arrive in one copy
        starts, at = [], 0
        for b in batch.nbytes:
            starts.append(at)
            at += (b // each + 31) // 32 * 32
        f, density, potential = (torch.zeros(at, device=DEV, dtype=fields[0].dtype) for _ in range(3))
        for s, x in zip(starts, fields):
            f[s:s + x.numel()] = x
        cut = lambda whole: [whole[s:s + b // each] for s, b in zip(starts, batch.nbytes)]  # noqa: E731
        phi = [p[:x.numel()].view(d) for p, x, d in zip(cut(potential), fields, dims)]
        state.update(batch=batch, f=f, density=density, ds=cut(density), ps=cut(potential), phi=phi)
    elif kind == "serve":
        dims = _dims_of(case)
        fields = _inputs(case, seed)
        torch.cuda.synchronize()
        state.update(server=ff.Server(4 << 30), phi=[torch.empty(d[:3], device=DEV, dtype=x.dtype)
                                                      for d, x in zip(dims, fields)],
                     requests=[(d[:3], x, _code(d[3])) for d, x in zip(dims, fields)])
    else:
        modes, phi = _inputs(case, seed)
        n = (case["ni"], case["nj"], case["nk"])
        state.update(n=n, modes=modes, phi=phi, precision=_code(case["precision"]),
                     f=torch.empty(n, device=DEV, dtype=phi.dtype))
    return state


def run(state):
    kind = state["kind"]
    if kind == "solve":
        state["into"].copy_(state["f"])
        state["plan"].solve(state["density"], state["whole"])
        return state["potential"]
    if kind == "plugin":
        state["into"].copy_(state["f"])
        stamps = []
        state["plan"].solve(state["plan"].bytes(), state["density"], state["whole"], stamps)
        return state["potential"]
    if kind == "batch":
        state["density"].copy_(state["f"])
        state["batch"].solve(state["ds"], state["ps"])
        return state["phi"]
    if kind == "serve":
        server = state["server"]
        ids = {server.submit(n, f, precision): q for q, (n, f, precision) in enumerate(state["requests"])}
        for _ in range(len(ids)):
            rid = server.next()[0]
            server.fetch(rid, state["phi"][ids[rid]])
        return state["phi"]
    ff.init_field(state["n"], state["f"], state["modes"], state["precision"])
    norms = ff.rel_norms(state["n"], state["phi"], state["modes"], state["precision"])
    return dict(f=state["f"], norms=norms)


# ------------------------------------------------- what a pass cannot do without
def work(case):
    if case["kind"] in ("solve", "plugin"):
        grids = [(case["ni"], case["nj"], case["nk"], case["precision"])]
    elif case["kind"] in ("batch", "serve"):
        grids = _dims_of(case)
    else:
        # the field written and phi read; per point the products and sums of
        # the analytic formulas, per mode one more cosine term (about 20
        # operations) in f and in both norms
        points = case["ni"] * case["nj"] * case["nk"]
        each = 8 if case["precision"] == "fp64" else 4
        return dict(bytes=2.0 * each * points, flops=points * (20.0 + 60.0 * case["modes"]))
    points = [(d[0] * d[1] * d[2], 8 if d[3] == "fp64" else 4) for d in grids]
    # f read and phi written; two real transforms (5/2 n log2 n each) and the filter
    return dict(bytes=float(sum(2 * p * e for p, e in points)),
                flops=float(sum(5 * p * math.log2(p) + 8 * p for p, _ in points)))


# ------------------------------------------------------- 64-bit values of the outputs
def _solve64(f, n):
    s = torch.fft.rfftn(f.view(n).double())
    # (min(i, n-i))^2 per axis: the reference domain's wavenumbers are whole
    k2 = None
    for axis, m in enumerate(n):
        q = torch.arange(s.shape[axis], device=DEV, dtype=torch.float64)
        q = torch.minimum(q, m - q) ** 2
        q = q.view([-1 if a == axis else 1 for a in range(3)])
        k2 = q if k2 is None else k2 + q
    k2 = k2.expand(s.shape).contiguous()
    k2[0, 0, 0] = 1.0
    s /= -k2
    s[0, 0, 0] = 0.0
    return torch.fft.irfftn(s, s=n)


def exact(case, seed):
    if case["kind"] in ("solve", "plugin"):
        return _solve64(_inputs(case, seed), (case["ni"], case["nj"], case["nk"]))
    if case["kind"] in ("batch", "serve"):
        return [_solve64(f, d[:3]) for f, d in zip(_inputs(case, seed), _dims_of(case))]
    n = (case["ni"], case["nj"], case["nk"])
    modes, phi = _inputs(case, seed)
    true = _analytic(n, modes, True).reshape(-1)
    d = (true - phi.double()).abs()
    norms = [float(d.sum() / true.abs().sum()), float(torch.sqrt(d.square().sum() / true.square().sum())),
             float(d.max() / true.abs().max())]
    return dict(f=_analytic(n, modes, False), norms=norms)
