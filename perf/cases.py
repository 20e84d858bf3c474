"""The work that a program using this engine has it do, as timed cases.

The spectral side is what the dycore calls every step: the transform pair, the
vorticity/divergence and wind pair, the gradient syntheses, the semi-implicit
solve, the whole step as one CUDA graph, and the ensemble batch.  The grid
side is the semi-Lagrangian gather and the departure search.  Sizes are those
of the benchmark configurations (T62, T126, T255 and T511, 40 levels, four or
five fields and ln ps, hence the odd plane counts) and of the tests (T21).

``exact`` is plain torch in 64 bits: the associated Legendre functions by
their three-term recurrence, dense per-order products, ``torch.fft``, and the
interpolation formulas written out.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
for _p in (str(ROOT), str(ROOT / "gpuwm-global_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

RADIUS = 6_371_220.0
DT = 300.0
F32, F64 = torch.float32, torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # One field at the smallest truncation in use: launches and host time.
        dict(name="pair_t21_f32_1", kind="pair", T=21, nlat=33, nlon=66, precision="float32", planes=1),
        # Double precision at T62, 40 levels x 4 fields + ln ps.
        dict(name="pair_t62_f64_161", kind="pair", T=62, nlat=94, nlon=192, precision="float64", planes=161),
        # The plain single-precision pair at T255, the same fields.
        dict(name="pair_t255_f32_161", kind="pair", T=255, nlat=384, nlon=768, precision="float32", planes=161),
        # T511, 40 levels x 5 fields: tensor cores, and the plain path beside them.
        dict(name="pair_t511_split_200", kind="pair", T=511, nlat=768, nlon=1536, precision="split16", planes=200),
        dict(name="pair_t511_f32_200", kind="pair", T=511, nlat=768, nlon=1536, precision="float32", planes=200),
        # The wind of 40 levels to vorticity and divergence and back.
        dict(name="vector_t511_split_40", kind="vector", T=511, nlat=768, nlon=1536, precision="split16", planes=40),
        # Synthesis of the wind and of the temperature and ln ps gradients.
        dict(name="synthesis_t255_f32_40", kind="synthesis", T=255, nlat=384, nlon=768, precision="float32", planes=40),
        # The semi-implicit solve of one step.
        dict(name="helmholtz_t255_f32_40", kind="helmholtz", T=255, nlat=384, nlon=768, precision="float32", planes=40),
        # Every transform of one dycore step, replayed as one graph.
        dict(name="step_t511_split_40", kind="step", T=511, nlat=768, nlon=1536, precision="split16", planes=40, fields=5),
        # 32 ensemble members and their control as one batch.
        dict(name="ensemble_t126_t255", kind="ensemble", T=126, nlat=192, nlon=384, precision="split16", planes=200, members=32),
        # Tracers read at departure points: 16 fields with the limiter.
        dict(name="gather_t511_f32_16", kind="gather", T=511, nlat=768, nlon=1536, precision="float32", planes=40, fields=16, order=4, limited=True),
        # The departure points of one step.
        dict(name="departure_t511_f32", kind="departure", T=511, nlat=768, nlon=1536, precision="float32", planes=40, iterations=3),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _smooth(n):
    """The next even number >= n with no prime factor above five."""
    n += n % 2
    while True:
        r = n
        for q in (2, 3, 5):
            while r % q == 0:
                r //= q
        if r == 1:
            return n
        n += 2


def draw(rng):
    kind = rng.choice(["pair", "pair", "pair", "vector", "synthesis", "helmholtz", "step", "ensemble",
                       "gather", "gather", "departure"])
    single = kind in ("step", "ensemble")
    precision = "split16" if single else rng.choice(["float32", "split16"])
    if kind in ("helmholtz", "gather", "departure"):
        precision = rng.choice(["float32", "float32", "float64"])
    elif kind == "pair":
        precision = rng.choice(["float32", "split16", "float64"])
    top = 255 if precision == "float64" else 511
    T = _log_int(rng, {"pair": 21, "ensemble": 42, "step": 126}.get(kind, 62), 126 if kind == "ensemble" else top)
    nlat, nlon = math.ceil(1.5 * (T + 1)), _smooth(3 * (T + 1))
    case = dict(kind=kind, T=T, nlat=nlat, nlon=nlon, precision=precision)
    room = (512 / (T + 1)) ** 2  # planes of this size to one of T511
    if kind == "pair":
        case["planes"] = _log_int(rng, 1, min(800, int(200 * room) if precision != "float64" else 200))
    elif kind in ("vector", "synthesis"):
        case["planes"] = _log_int(rng, 1, 60)
    elif kind in ("helmholtz", "departure"):
        case["planes"] = rng.randint(10, 60)
    elif kind == "step":
        case.update(planes=rng.randint(10, 40), fields=rng.randint(1, 5))
    elif kind == "ensemble":
        case.update(planes=rng.randint(20, 200), members=rng.randint(2, 32))
    if kind == "departure":
        case["iterations"] = rng.randint(2, 4)
    if kind == "gather":
        case.update(planes=rng.randint(10, 40), fields=rng.randint(1, 16), order=rng.choice([4, 4, 6]))
        case["limited"] = case["order"] == 4 and rng.random() < 0.6
        if case["order"] == 6:
            case["fields"] = min(case["fields"], 6)
    return case


def _control(case):
    """The control's grid of an ensemble: twice the members' resolution."""
    T = 2 * case["T"] + 1
    if case["nlon"] == 384:
        return T, 384, 768
    return min(T, 255), math.ceil(1.5 * (min(T, 255) + 1)), _smooth(3 * (min(T, 255) + 1))


# --------------------------------------------------- plain 64-bit mathematics
@functools.lru_cache(maxsize=8)
def _nodes(n):
    """Gauss nodes (ascending) and weights, by Newton's iteration in extended
    precision."""
    x = np.cos(np.pi * (np.arange(n, dtype=np.longdouble) + np.longdouble(0.75)) / (n + np.longdouble(0.5)))
    for _ in range(8):
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
        dp = n * (x * p1 - p0) / (x * x - 1)
        x = x - p1 / dp
    w = 2 / ((1 - x * x) * dp * dp)
    return x[::-1].astype(np.float64), w[::-1].astype(np.float64)


def _sphere(case):
    mu, w = (torch.as_tensor(v.copy(), device="cuda") for v in _nodes(case["nlat"]))
    return mu, w, torch.sqrt((1 - mu) * (1 + mu))


@functools.lru_cache(maxsize=2)
def _legendre(T, nlat):
    """Orthonormal P_nm at the Gauss latitudes, (m, n, lat)."""
    mu, _, cos = _sphere(dict(nlat=nlat))
    m = torch.arange(T + 1, dtype=F64, device="cuda")[:, None]
    p = torch.zeros(T + 1, T + 1, nlat, dtype=F64, device="cuda")
    seed = torch.full((nlat,), math.sqrt(0.25 / math.pi), dtype=F64, device="cuda")
    p[0, 0] = seed
    for k in range(1, T + 1):
        seed = seed * cos * -math.sqrt((2 * k + 1) / (2 * k))
        p[k, k] = seed
    eps = lambda n: torch.sqrt((n * n - m * m).clamp(min=0) / (4 * n * n - 1))  # noqa: E731
    for n in range(1, T + 1):
        old = eps(n - 1) * p[:, n - 2] if n > 1 else 0.0
        new = (mu * p[:, n - 1] - old) / eps(n)
        p[:n, n] = new[:n]
    return p


@functools.lru_cache(maxsize=1)
def _slope(T, nlat):
    """d P_nm / d latitude, (m, n, lat)."""
    mu, _, cos = _sphere(dict(nlat=nlat))
    p = _legendre(T, nlat)
    m = torch.arange(T + 1, dtype=F64, device="cuda")[:, None]
    d = torch.zeros_like(p)
    for n in range(1, T + 1):
        eps = torch.sqrt((n * n - m * m).clamp(min=0) / (4 * n * n - 1))
        d[:, n] = ((2 * n + 1) * eps * p[:, n - 1] - n * mu * p[:, n]) / cos
    return d


def _to_waist(table, c):
    """sum_n table[m, n, lat] c[plane, n, m] -> (plane, lat, m)."""
    x = torch.view_as_real(c.permute(2, 1, 0).contiguous()).flatten(2)
    y = torch.bmm(table.transpose(1, 2), x)
    return torch.view_as_complex(y.unflatten(2, (-1, 2)).contiguous()).permute(2, 1, 0)


def _from_waist(table, weight, f):
    """sum_lat weight[lat] table[m, n, lat] f[plane, lat, m] -> (plane, n, m)."""
    x = torch.view_as_real((f * weight[:, None]).permute(2, 1, 0).contiguous()).flatten(2)
    y = torch.bmm(table, x)
    c = torch.view_as_complex(y.unflatten(2, (-1, 2)).contiguous()).permute(2, 1, 0).contiguous()
    c[..., 0].imag.zero_()
    return c


def _grid(w, nlon):
    return torch.fft.irfft(w, n=nlon, dim=-1, norm="forward")


def _planewise(f, *xs, step=200):
    """f over slices of the leading axis, the results put together."""
    parts = [f(*(x[k:k + step] for x in xs)) for k in range(0, xs[0].shape[0], step)]
    if isinstance(parts[0], tuple):
        return tuple(torch.cat(p) for p in zip(*parts))
    return torch.cat(parts)


def _inverse(c, nlat, nlon):
    return _planewise(lambda x: _grid(_to_waist(_legendre(c.shape[-1] - 1, nlat), x), nlon), c)


def _forward(g, T):
    nlat, nlon = g.shape[-2:]
    _, w, _ = _sphere(dict(nlat=nlat))
    return _planewise(lambda x: _from_waist(_legendre(T, nlat), 2 * math.pi * w,
                                            torch.fft.rfft(x, dim=-1)[..., :T + 1] / nlon), g)


def _im(T):
    return 1j * torch.arange(T + 1, dtype=F64, device="cuda")


def _gradient(c, nlat, nlon):
    T = c.shape[-1] - 1
    _, _, cos = _sphere(dict(nlat=nlat))
    east = _grid(_to_waist(_legendre(T, nlat), c * _im(T)), nlon) / (RADIUS * cos[:, None])
    return east, _grid(_to_waist(_slope(T, nlat), c), nlon) / RADIUS


def _wind(z, d, nlat, nlon):
    n = torch.arange(z.shape[-1], dtype=F64, device="cuda")[:, None]
    inv = torch.where(n > 0, -RADIUS ** 2 / (n * (n + 1)).clamp(min=1), 0.0)
    pe, pn = _gradient(z * inv, nlat, nlon)
    ce, cn = _gradient(d * inv, nlat, nlon)
    return ce - pn, pe + cn


def _vordiv(u, v, T):
    nlat, nlon = u.shape[-2:]
    _, w, cos = _sphere(dict(nlat=nlat))
    fu, fv = (torch.fft.rfft(x, dim=-1)[..., :T + 1] / nlon for x in (u, v))
    rot = lambda f: _from_waist(_legendre(T, nlat), 2 * math.pi * w / (RADIUS * cos), f * _im(T))  # noqa: E731
    shear = lambda f: _from_waist(_slope(T, nlat), 2 * math.pi * w / RADIUS, f)  # noqa: E731
    return rot(fv) + shear(fu), rot(fu) - shear(fv)


def _solve(b, c, tau, div, theta, lnps):
    """(I - tau L) y = r per degree: D' and x' = x + tau C D'."""
    T = div.shape[-1] - 1
    b, c = (torch.as_tensor(x, device="cuda") for x in (b, c))
    n = torch.arange(T + 1, dtype=F64, device="cuda")
    k2 = n * (n + 1) / RADIUS ** 2
    x = torch.cat([theta, lnps[None]])
    real = lambda a: torch.view_as_real(a.permute(1, 0, 2).contiguous()).flatten(2)  # noqa: E731
    back = lambda a: torch.view_as_complex(a.unflatten(2, (-1, 2)).contiguous()).permute(1, 0, 2)  # noqa: E731
    rhs = real(div) + tau * k2[:, None, None] * (b @ real(x))
    m = torch.eye(b.shape[0], dtype=F64, device="cuda") - tau ** 2 * k2[:, None, None] * (b @ c)
    d = torch.linalg.solve(m, rhs)
    d[0] = real(div)[0]
    y = real(x) + tau * (c @ d)
    y[0] = real(x)[0]
    y = back(y)
    return back(d).contiguous(), y[:-1].contiguous(), y[-1].contiguous()


def _rows(case, half):
    """Latitudes with `half` rows reflected beyond each pole, the row each one
    reads, and whether it reads it half a turn round."""
    lat = torch.asin(_sphere(case)[0])
    nj = case["nlat"]
    k = torch.arange(half, device="cuda")
    south, north = k.flip(0), nj - 1 - k
    ext = torch.cat([-math.pi - lat[south], lat, math.pi - lat[north]])
    row = torch.cat([south, torch.arange(nj, device="cuda"), north])
    turned = torch.cat([k * 0 + 1, torch.zeros(nj, dtype=k.dtype, device="cuda"), k * 0 + 1])
    return ext, row, turned


def _lagrange(x, nodes):
    w = []
    for a in range(len(nodes)):
        t = torch.ones_like(x)
        for b in range(len(nodes)):
            if b != a:
                t = t * (x - nodes[b]) / (nodes[a] - nodes[b])
        w.append(t)
    return w


def _interpolate(case, f, xi, phi, lev):
    """The gather of f (fields, nk, nj, ni) at points of any shape."""
    nh, nk, ni = case["order"], f.shape[1], f.shape[3]
    g = nh // 2 - 1
    ext, row, turned = _rows(case, nh // 2)
    flat = f.reshape(f.shape[0], -1)
    p = phi.clamp(-math.pi / 2, math.pi / 2)
    s = (torch.searchsorted(ext, p, right=True) - 1).clamp(g, case["nlat"] + g) - g
    z = lev.clamp(-0.5, nk - 0.5)
    kb = torch.floor(z).long().clamp(0, nk - 2)
    k0 = (kb - 1).clamp(0, nk - 4)
    i0 = torch.floor(xi).long() - g
    wx = _lagrange(xi - i0, [torch.full_like(xi, float(q)) for q in range(nh)])
    wy = _lagrange(p, [ext[s + m] for m in range(nh)])
    wz = _lagrange(z - k0, [torch.full_like(z, float(q)) for q in range(4)])
    level, lo, hi = [], None, None
    for c in range(4):
        total = 0.0
        for m in range(nh):
            base = ((k0 + c) * case["nlat"] + row[s + m]) * ni
            for q in range(nh):
                v = flat[:, base + (i0 + q + turned[s + m] * (ni // 2)) % ni]
                total = total + (wx[q] * wy[m]) * v
                if case["limited"] and m in (g, g + 1) and q in (g, g + 1):
                    cell = (k0 + c == kb) | (k0 + c == kb + 1)
                    low, high = torch.where(cell, v, math.inf), torch.where(cell, v, -math.inf)
                    lo = low if lo is None else torch.minimum(lo, low)
                    hi = high if hi is None else torch.maximum(hi, high)
        level.append(total)
    r = sum(w * t for w, t in zip(wz, level))
    if case["limited"]:
        return torch.minimum(torch.maximum(r, lo), hi)
    edge, near = torch.where(z < 0, level[0], level[3]), torch.where(z < 0, level[1], level[2])
    face = edge + 0.5 * (edge - near)
    held = torch.minimum(torch.maximum(r, torch.minimum(edge, face)), torch.maximum(edge, face))
    return torch.where((z < 0) | (z > nk - 1), held, r)


def _linear(case, f, q, k):
    """The wind f (4, nk, nj, ni) at the points q (3, ...) of the unit sphere."""
    nk, ni = f.shape[1], f.shape[3]
    ext, row, turned = _rows(case, 2)
    flat = f.reshape(4, -1)
    phi = torch.atan2(q[2], torch.hypot(q[0], q[1]))
    x = torch.atan2(q[1], q[0]) * (ni / (2 * math.pi))
    s = (torch.searchsorted(ext, phi, right=True) - 1).clamp(1, case["nlat"] + 1)
    z = k.clamp(0, nk - 1)
    k0 = torch.floor(z).long().clamp(0, nk - 2)
    i0 = torch.floor(x).long()
    ax, ay, az = x - i0, (phi - ext[s]) / (ext[s + 1] - ext[s]), z - k0
    out = 0.0
    for c, wc in ((0, 1 - az), (1, az)):
        for m, wm in ((0, 1 - ay), (1, ay)):
            for e, we in ((0, 1 - ax), (1, ax)):
                col = (i0 + e + turned[s + m] * (ni // 2)) % ni
                out = out + (wc * wm * we) * flat[:, ((k0 + c) * case["nlat"] + row[s + m]) * ni + col]
    return out


def _arrivals(case):
    mu, _, cos = _sphere(case)
    lon = torch.arange(case["nlon"], dtype=F64, device="cuda") * (2 * math.pi / case["nlon"])
    return torch.stack([cos[:, None] * torch.cos(lon), cos[:, None] * torch.sin(lon), mu[:, None].expand(-1, len(lon))])


def _departures(case, wind, ahead, iterations):
    """Fixed-point search in 64 bits: coordinates per level and the largest
    moves and displacements."""
    a, ni, out, most = _arrivals(case), case["nlon"], [], []
    lat = torch.asin(_sphere(case)[0])
    ext = _rows(case, 2)[0]
    cell = (RADIUS * 0.5 * (ext[3:-1] - ext[1:-3]))[:, None]
    top = case["planes"] - 0.5
    unit = lambda v: v / v.norm(dim=0)  # noqa: E731
    for k in range(case["planes"]):
        here, there = wind[:, k], ahead[:, k]
        q, z = unit(a - DT / RADIUS * here[:3]), (k - DT * here[3]).clamp(-0.5, top)
        for _ in range(iterations):
            w = _linear(case, wind, q, z) + there
            p, y = unit(a - 0.5 * DT / RADIUS * w[:3]), (k - 0.5 * DT * w[3]).clamp(-0.5, top)
            move, lift, q, z = 2 * RADIUS * torch.asin(0.5 * (p - q).norm(dim=0)), (y - z).abs(), p, y
        xi, phi = torch.atan2(q[1], q[0]) * (ni / (2 * math.pi)), torch.atan2(q[2], torch.hypot(q[0], q[1]))
        far = 2 * RADIUS * torch.asin((0.5 * (q - a).norm(dim=0)).clamp(max=1))
        out.append(torch.stack([xi, phi, z]))
        most.append(torch.stack([move.max(), (move / cell).max(), lift.max(), far.max(), (far / cell).max(), (z - k).abs().max()]))
    return torch.stack(out, dim=1), torch.stack(most).amax(dim=0)


# ------------------------------------------------------------------ the inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _red(T, planes, g, power=1.5):
    """Red-spectrum coefficients (planes, n, m) with unit total variance."""
    n = torch.arange(T + 1, dtype=F64, device="cuda")
    sigma = torch.where(n > 0, (n * (n + 1)).clamp(min=1) ** -power, 0.0)[:, None]
    c = torch.complex(*(torch.randn((planes, T + 1, T + 1), generator=g, device="cuda", dtype=F64) for _ in "ri"))
    c = torch.tril(c * sigma)
    c[..., 0].imag.zero_()
    return c / math.sqrt(float((2 * (2 * n + 1) * sigma[:, 0] ** 2).sum()) / (4 * math.pi))


def _field(case, planes, g, dtype, mean=0.0, spread=1.0):
    """A red-spectrum field (planes, nlat, nlon)."""
    out = torch.empty(planes, case["nlat"], case["nlon"], dtype=dtype, device="cuda")
    for k in range(0, planes, 200):
        c = _red(case["T"], min(200, planes - k), g)
        out[k:k + 200] = mean + spread * _inverse(c, case["nlat"], case["nlon"])
    return out


def _flow(case, g, dtype):
    """Cartesian wind (m/s) and level rate (levels/s), (4, nlev, nlat, nlon)."""
    L = case["planes"]
    a = _arrivals(case)
    east, north = _field(case, L, g, F64, spread=25.0), _field(case, L, g, F64, spread=12.0)
    mu, _, cos = _sphere(case)
    east = (east + 20.0) * cos[:, None]  # single-valued at the poles
    north = north * cos[:, None]
    lon = a[:2] / cos[:, None]
    v = [-east * lon[1] - north * mu[:, None] * lon[0], east * lon[0] - north * mu[:, None] * lon[1], north * cos[:, None],
         _field(case, L, g, F64, spread=1e-3)]
    return torch.stack([x.to(dtype) for x in v])


def _dtype(case):
    return F64 if case["precision"] == "float64" else F32


@functools.lru_cache(maxsize=2)
def _transform(T, nlat, nlon, precision):
    """The plan that a program makes once and keeps."""
    from b200sht import SphericalHarmonicTransform

    # T62 is run on 94 rows, one under the three-halves rule
    dealias = min(1.5, (nlat - 0.5) / (T + 1))
    return SphericalHarmonicTransform.create(T, nlat=nlat, nlon=nlon, precision=precision, dealias_factor=dealias)


@functools.lru_cache(maxsize=2)
def _tables(T, nlat, nlon, precision):
    from b200sht import GaussianGrid
    from b200sht.semilag import SphericalGridTables

    return SphericalGridTables.create(GaussianGrid.create(T, nlat=nlat, nlon=nlon), dtype=F64 if precision == "float64" else F32)


def _plan_key(case):
    return case["T"], case["nlat"], case["nlon"], case["precision"]


def _vertical(nlev):
    from b200sht.semi_implicit import VerticalModeOperator
    from b200sht.synthetic import seeded_vertical_operator

    b, c = seeded_vertical_operator(nlev)
    return VerticalModeOperator(b, c), b, c


def _inputs(case, seed):
    """The arrays a case starts from, by name."""
    g, kind, dt = _generator(seed), case["kind"], _dtype(case)
    T, P = case["T"], case["planes"]
    cdt = torch.complex128 if dt == F64 else torch.complex64
    if kind == "pair":
        return dict(grid=_field(case, P, g, dt, 250.0, 20.0))
    if kind == "vector":
        u, v = _wind(1e-5 * _red(T, P, g, 1.0), 1e-6 * _red(T, P, g, 1.0), case["nlat"], case["nlon"])
        return dict(u=u.to(dt), v=v.to(dt))
    if kind == "synthesis":
        return dict(vorticity=(1e-5 * _red(T, P, g, 1.0)).to(cdt), divergence=(1e-6 * _red(T, P, g, 1.0)).to(cdt),
                    theta=(20.0 * _red(T, P, g)).to(cdt), lnps=(0.1 * _red(T, 1, g))[0].to(cdt))
    if kind == "helmholtz":
        return dict(divergence=(1e-6 * _red(T, P, g, 1.0)).to(cdt), theta=(20.0 * _red(T, P, g)).to(cdt), lnps=(0.1 * _red(T, 1, g))[0].to(cdt))
    if kind == "step":
        u, v = _wind(1e-5 * _red(T, P, g, 1.0), 1e-6 * _red(T, P, g, 1.0), case["nlat"], case["nlon"])
        scalars = _field(case, case["fields"] * P, g, dt, 250.0, 20.0).unflatten(0, (case["fields"], P))
        return dict(scalars=scalars, lnps=_field(case, 1, g, dt, 11.5, 0.1)[0], u=u.to(dt), v=v.to(dt))
    if kind == "ensemble":
        T2, nlat2, nlon2 = _control(case)
        control = dict(case, T=T2, nlat=nlat2, nlon=nlon2)
        members = _field(case, case["members"] * P, g, dt, 250.0, 20.0)
        return dict(members=members, control=_field(control, P, g, dt, 250.0, 20.0))
    if kind == "gather":
        flow = _flow(case, g, F64)
        k = torch.arange(P, dtype=F64, device="cuda")[:, None, None]
        q = _arrivals(case)[:, None] - DT / RADIUS * flow[:3]
        xi = torch.atan2(q[1], q[0]) * (case["nlon"] / (2 * math.pi))
        phi = torch.atan2(q[2], torch.hypot(q[0], q[1]))
        return dict(xi=xi.to(dt), phi=phi.to(dt), level=(k - DT * flow[3]).to(dt),
                    fields=[_field(case, P, g, dt, 5.0, 2.0) for _ in range(case["fields"])])
    return dict(wind=_flow(case, g, dt), ahead=_flow(case, g, dt))


def prepare(case, seed):
    from b200sht import VorticityDivergenceOperator
    from b200sht.batch import TransformBatch
    from b200sht.semi_implicit import VerticalModeSemiImplicit
    from b200sht.semilag import CartesianWind, Stencil
    from b200sht.step import DycoreTransformStep
    from b200sht.transform import SphericalHarmonicTransform

    kind, x = case["kind"], _inputs(case, seed)
    s = dict(case=case, x=x)
    if kind in ("pair", "vector", "synthesis", "helmholtz"):
        s["t"] = _transform(*_plan_key(case))
        s["vector"] = VorticityDivergenceOperator(s["t"])
    if kind == "helmholtz":
        s["solver"], s["vertical"] = VerticalModeSemiImplicit(), _vertical(case["planes"])[0]
    elif kind == "step":
        # a graph holds its plan's buffers, so the step has a plan of its own
        T, nlat, nlon, precision = _plan_key(case)
        t = SphericalHarmonicTransform.create(T, nlat=nlat, nlon=nlon, precision=precision)
        s["step"] = DycoreTransformStep(t, _vertical(case["planes"])[0], n_scalar=case["fields"], dt_s=DT)
        s["step"].load(**x)
        s["step"].capture()
        s["step"].load(**x)
    elif kind == "ensemble":
        T2, nlat2, nlon2 = _control(case)
        plans = [_transform(*_plan_key(case)), _transform(T2, nlat2, nlon2, case["precision"])]
        s["batch"] = TransformBatch(plans, [case["members"] * case["planes"], case["planes"]])
    elif kind == "gather":
        s["stencil"] = Stencil(xi=x["xi"], phi=x["phi"], level=x["level"], tables=_tables(*_plan_key(case)))
    elif kind == "departure":
        s["tables"] = _tables(*_plan_key(case))
        s["wind"], s["ahead"] = CartesianWind(*x["wind"]), CartesianWind(*x["ahead"])
    return s


def run(s):
    from b200sht.semilag import departure_points, gather_batch

    case, x = s["case"], s["x"]
    kind = case["kind"]
    if kind == "pair":
        coeff = s["t"].forward(x["grid"])
        return dict(coeff=coeff, grid=s["t"].inverse(coeff))
    if kind == "vector":
        zeta, div = s["vector"].vordiv_from_wind(x["u"], x["v"])
        u, v = s["vector"].wind_from_vordiv(zeta, div)
        return dict(vorticity=zeta, divergence=div, u=u, v=v)
    if kind == "synthesis":
        u, v = s["vector"].wind_from_vordiv(x["vorticity"], x["divergence"])
        te, tn = s["t"].gradient(x["theta"])
        pe, pn = s["t"].gradient(x["lnps"])
        return dict(u=u, v=v, theta_east=te, theta_north=tn, lnps_east=pe, lnps_north=pn)
    if kind == "helmholtz":
        d, th, lp = s["solver"].solve_arrays(s["t"], s["vertical"], 0.5 * DT, x["divergence"], x["theta"], x["lnps"])
        return dict(divergence=d, theta=th, lnps=lp)
    if kind == "step":
        st = s["step"]
        st.replay()
        return dict(scalars=st.scalar_coeff, lnps=st.lnps_coeff, vorticity=st.vorticity, divergence=st.div_solved, theta=st.theta_solved,
                    lnps_new=st.lnps_solved, u=st.u, v=st.v, grad_theta=st.grad_theta, grad_lnps=st.grad_lnps, div_grid=st.div_grid)
    if kind == "ensemble":
        coeffs = s["batch"].forward([x["members"], x["control"]])
        return dict(coeffs=coeffs, grids=s["batch"].inverse(coeffs))
    if kind == "gather":
        return dict(values=gather_batch(x["fields"], s["stencil"], monotone=case["limited"], order=case["order"]))
    stencil, most = departure_points(s["wind"], s["tables"], DT, iterations=case["iterations"], extrapolated=s["ahead"])
    most = [most.move_max_m, most.move_max_cells, most.move_max_levels, most.displacement_max_m, most.displacement_max_cells, most.displacement_max_levels]
    return dict(xi=stencil.xi, phi=stencil.phi, level=stencil.level, most=np.array(most))


def exact(case, seed):
    x, kind, T = _inputs(case, seed), case["kind"], case["T"]
    nlat, nlon = case["nlat"], case["nlon"]
    wide = lambda a: a.to(torch.complex128 if a.is_complex() else F64)  # noqa: E731
    if kind == "pair":
        coeff = _forward(wide(x["grid"]), T)
        return dict(coeff=coeff, grid=_inverse(coeff, nlat, nlon))
    if kind == "vector":
        zeta, div = _vordiv(wide(x["u"]), wide(x["v"]), T)
        u, v = _wind(zeta, div, nlat, nlon)
        return dict(vorticity=zeta, divergence=div, u=u, v=v)
    if kind == "synthesis":
        u, v = _wind(wide(x["vorticity"]), wide(x["divergence"]), nlat, nlon)
        te, tn = _gradient(wide(x["theta"]), nlat, nlon)
        pe, pn = _gradient(wide(x["lnps"])[None], nlat, nlon)
        return dict(u=u, v=v, theta_east=te, theta_north=tn, lnps_east=pe[0], lnps_north=pn[0])
    if kind == "helmholtz":
        _, b, c = _vertical(case["planes"])
        return dict(zip(("divergence", "theta", "lnps"), _solve(b, c, 0.5 * DT, wide(x["divergence"]), wide(x["theta"]), wide(x["lnps"]))))
    if kind == "step":
        _, b, c = _vertical(case["planes"])
        scalars = _forward(wide(x["scalars"]).flatten(0, 1), T).unflatten(0, (case["fields"], -1))
        lnps = _forward(wide(x["lnps"])[None], T)[0]
        zeta, div = _vordiv(wide(x["u"]), wide(x["v"]), T)
        d, th, lp = _solve(b, c, 0.5 * DT, div, scalars[0], lnps)
        u, v = _wind(zeta, d, nlat, nlon)
        return dict(scalars=scalars, lnps=lnps, vorticity=zeta, divergence=d, theta=th, lnps_new=lp, u=u, v=v,
                    grad_theta=torch.stack(_gradient(th, nlat, nlon)), grad_lnps=torch.stack([y[0] for y in _gradient(lp[None], nlat, nlon)]),
                    div_grid=_inverse(d, nlat, nlon))
    if kind == "ensemble":
        T2, nlat2, nlon2 = _control(case)
        coeffs = [_forward(wide(x["members"]), T), _forward(wide(x["control"]), T2)]
        return dict(coeffs=coeffs, grids=[_inverse(coeffs[0], nlat, nlon), _inverse(coeffs[1], nlat2, nlon2)])
    if kind == "gather":
        f = torch.stack([wide(a) for a in x["fields"]])
        out = torch.empty_like(f)
        for k in range(case["planes"]):
            out[:, k] = _interpolate(case, f, *(wide(x[n][k]) for n in ("xi", "phi", "level")))
        return dict(values=list(out))
    at, most = _departures(case, wide(x["wind"]), wide(x["ahead"]), case["iterations"])
    return dict(xi=at[0], phi=at[1], level=at[2], most=most.cpu().numpy())


# ------------------------------------------------------------- work, tolerance
def work(case):
    """Inputs and outputs once; multiplications and additions of the folded
    triangle, the FFTs, the vertical products or the interpolation."""
    kind, T, P = case["kind"], case["T"], case["planes"]
    size = 8 if case["precision"] == "float64" else 4
    points = case["nlat"] * case["nlon"]

    def one(T, nlat, nlon):  # bytes of a grid and of a spectrum, operations of one transform
        return size * nlat * nlon, size * (T + 1) * (T + 2), nlat * (T + 1) * (T + 2) + 2.5 * nlat * nlon * math.log2(nlon)

    grid, spec, ops = one(T, case["nlat"], case["nlon"])
    solve = 4 * P * (4 * P + 2) * (T + 1) * (T + 2) / 2
    if kind == "pair":
        return dict(bytes=2 * P * (grid + spec), flops=2 * P * ops)
    if kind == "vector":
        return dict(bytes=4 * P * (grid + spec), flops=8 * P * ops)
    if kind == "synthesis":
        return dict(bytes=P * (2 * spec + 2 * grid) + (P + 1) * (spec + 2 * grid), flops=(4 * P + 2 * (P + 1)) * ops)
    if kind == "helmholtz":
        return dict(bytes=2 * (2 * P + 1) * spec, flops=solve)
    if kind == "step":
        n = case["fields"] * P + 1
        return dict(bytes=n * (grid + spec) + 2 * P * (grid + spec) + 2 * (2 * P + 1) * spec + P * grid + 2 * P * grid + 2 * (P + 1) * grid,
                    flops=(n + 4 * P + P + 4 * P + 2 * (P + 1)) * ops + solve)
    if kind == "ensemble":
        grid2, spec2, ops2 = one(*_control(case))
        return dict(bytes=2 * P * (case["members"] * (grid + spec) + grid2 + spec2), flops=2 * P * (case["members"] * ops + ops2))
    n = P * points
    if kind == "gather":
        return dict(bytes=size * n * (3 + 2 * case["fields"]), flops=n * case["fields"] * 3 * 4 * case["order"] ** 2)
    return dict(bytes=size * n * (8 + 3), flops=n * case["iterations"] * 150)


def tolerance(case):
    """About four times the error against ``exact``.  The divergence of a
    nearly rotational wind, and the gradient of ln ps beside its mean, lose
    digits to cancellation in any 32-bit transform; a 32-bit departure point
    beside the date line may fall on either side of it."""
    if case["precision"] == "float64":
        return {"rel": 2e-13 if case["kind"] == "departure" else 1e-13}
    if case["kind"] == "step":
        return {"rel": 0.03}
    return {"rel": dict(pair=3e-6, vector=5e-4, synthesis=2e-6, helmholtz=2e-6, ensemble=2e-6, gather=8e-5, departure=6e-3)[case["kind"]]}
