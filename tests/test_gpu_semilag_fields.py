"""Gathers of several separate fields (interleaved in groups of 16 bytes, the
rest in a pair and a single) against the one-field call, and the departure
search's diagnostics against its move arrays."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(dtype, nlat=37, nlon=74, nlev=7):
    import torch

    from b200sht import GaussianGrid
    from b200sht.semilag import SphericalGridTables
    from b200sht.workloads import rotation_departures

    grid = GaussianGrid.create(21, nlat=nlat, nlon=nlon)
    tables = SphericalGridTables.create(grid, dtype=dtype)
    xi, phi, lev = rotation_departures(grid.lat_rad, nlon, nlev, speed=400.0, dtype=dtype)
    gen = torch.Generator(device="cuda").manual_seed(3)
    field = lambda: torch.randn((nlev, nlat, nlon), generator=gen, device="cuda", dtype=dtype)  # noqa: E731
    return tables, (xi, phi, lev), field


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("kw", [dict(monotone=True), dict(monotone=False),
                                dict(monotone=False, order=6), dict(monotone=True, order=6),
                                dict(monotone=True, deficit=True)])
def test_grouped_fields_equal_single_fields(dtype, kw):
    import torch

    from b200sht.semilag import Stencil, gather_batch

    tables, at, field = _setup(getattr(torch, dtype))
    st = Stencil(*at, tables=tables)
    fields = [field() for _ in range(19)]
    fields[2] = fields[2].transpose(1, 2).contiguous().transpose(1, 2)  # not contiguous
    single = [gather_batch([f], st, **kw)[0] for f in fields]
    flat = lambda r: r if isinstance(r, tuple) else (r,)  # noqa: E731
    for count, batch in ((2, 16), (3, 16), (4, 16), (5, 16), (7, 16), (19, 19), (19, 6)):
        got = gather_batch(fields[:count], st, batch=batch, **kw)
        for a, b in zip(got, single):
            assert all(torch.equal(x, y) for x, y in zip(flat(a), flat(b)))
    band = tables.window(slice(4, 30), slice(9, 24))
    held = [f[:, 4:30].contiguous() for f in fields[:7]]
    st = Stencil(*(x[:, 9:24].contiguous() for x in at), tables=tables, window=band)
    for a, b in zip(gather_batch(held, st, **kw), single):
        assert all(torch.equal(x, y[:, 9:24]) for x, y in zip(flat(a), flat(b)))


@pytest.mark.parametrize("dtype, tol", [("float64", 1e-11), ("float32", 2e-4)])
@pytest.mark.parametrize("solver", ["fixed_point", "newton", "newton_ls"])
def test_search_maxima_match_the_move_arrays(dtype, tol, solver):
    """The maxima of the moves the arrays hold, and the displacement as a
    great-circle distance in float64 (float32: a unit vector's rounding,
    6e-8 rad, against displacements of a few 1e-3 rad)."""
    import torch

    from b200sht.semilag import (CartesianWind, departure_points, meridional_grid_length_m,
                                 search_into)

    dt = getattr(torch, dtype)
    tables, _, field = _setup(dt)
    wind = [30.0 * field() for _ in range(3)] + [1e-3 * field()]
    ahead = [30.0 * field() for _ in range(3)] + [1e-3 * field()]
    outs = [torch.empty_like(wind[0]) for _ in range(5)]
    search_into(tables, wind + ahead, 3, 300.0, outs, solver=solver)
    st, d = departure_points(CartesianWind(*wind), tables, 300.0, extrapolated=CartesianWind(*ahead),
                             solver=solver)
    assert all(torch.equal(a, b) for a, b in zip((st.xi, st.phi, st.level), outs))
    xi, phi, lev, move_m, move_k = (x.double().cpu().numpy() for x in outs)
    cell = meridional_grid_length_m(tables)[None, :, None]
    lat = tables.host_tables(4)["lat_ext"][2:-2][None, :, None]
    dlam = 2 * np.pi / tables.nlon
    dl = (xi - np.arange(tables.nlon)) * dlam
    hav = np.sin(0.5 * (phi - lat)) ** 2 + np.cos(lat) * np.cos(phi) * np.sin(0.5 * dl) ** 2
    dist = 2 * tables.radius_m * np.arcsin(np.sqrt(hav))
    want = [move_m.max(), (move_m / cell).max(), move_k.max(), dist.max(), (dist / cell).max(),
            np.abs(lev - np.arange(lev.shape[0])[:, None, None]).max()]
    got = [d.move_max_m, d.move_max_cells, d.move_max_levels, d.displacement_max_m,
           d.displacement_max_cells, d.displacement_max_levels]
    np.testing.assert_allclose(got, want, rtol=tol)
    # a NaN level rate is clamped to the lowest interface, no NaN in any level
    wind[3][2, 5, 6] = float("nan")
    st, d = departure_points(CartesianWind(*wind), tables, 300.0, solver=solver)
    assert float(st.level[2, 5, 6]) == -0.5 and not bool(torch.isnan(st.level).any())
    assert 2.5 <= d.displacement_max_levels < lev.shape[0]
    # a NaN horizontal wind leaves the displacement NaN, whatever the solver,
    # and the last move only where the line search reports the step at the point
    wind[0][3, 9, 12] = float("nan")
    st, d = departure_points(CartesianWind(*wind), tables, 300.0, solver=solver)
    assert bool(torch.isnan(st.xi[3, 9, 12])) and bool(torch.isnan(st.phi[3, 9, 12]))
    assert np.isnan(d.displacement_max_m) and np.isnan(d.displacement_max_cells)
    assert np.isnan(d.move_max_m) == np.isnan(d.move_max_cells) == (solver == "newton_ls")
    assert np.isfinite([d.move_max_levels, d.displacement_max_levels]).all()


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("ahead", [False, True])
def test_a_wind_that_is_not_finite_stays_at_its_points(dtype, bad, ahead):
    """One horizontal component of the advecting or the extrapolated wind not
    finite at one point: NaN where its value is read (the point itself, and
    the points whose taps hold it), every other point as without it, on the
    whole grid and on a band that holds every row (a NaN latitude counts as
    the south pole's, so a smaller one escapes)."""
    import torch

    from b200sht.semilag import CartesianWind, departure_points

    tables, _, field = _setup(getattr(torch, dtype))
    wind, ex = ([30.0 * field() for _ in range(3)] + [1e-3 * field()] for _ in range(2))
    search = lambda **kw: departure_points(CartesianWind(*wind), tables, 300.0,  # noqa: E731
                                           extrapolated=CartesianWind(*ex), **kw)
    clean, _ = search()
    at = (3, 20, 70)
    part = (ex if ahead else wind)[1]
    keep, part[at] = part[at].clone(), 60.0
    other, _ = search()  # another finite value: what moves reads the point
    part[at] = bad
    band = tables.window(slice(0, tables.nlat), slice(0, tables.nlat))
    for kw in (dict(), dict(window=band, defer_escape=True)):
        got, d = search(**kw)
        lost = torch.isnan(got.xi)
        assert lost[at] and int(lost.sum()) <= (1 if ahead else 64)
        assert torch.equal(lost, torch.isnan(got.phi))
        moved = (other.xi != clean.xi) | (other.phi != clean.phi)
        assert bool((lost | ~moved).all())
        for name in ("xi", "phi", "level"):
            assert torch.equal(getattr(got, name)[~lost], getattr(clean, name)[~lost])
        assert np.isnan(d.displacement_max_m) and np.isnan(d.displacement_max_cells)
        assert np.isfinite([d.move_max_m, d.move_max_levels, d.displacement_max_levels]).all()
    part[at] = keep


@pytest.mark.parametrize("shape", [(131074, 4, 6), (4, 131074, 6)])
def test_more_levels_or_rows_than_a_grid_dimension(shape):
    """Levels and rows past 65535 blocks, where a call takes several launches:
    a resting wind departs from its arrival points, and the gather there
    returns the field bit for bit."""
    import types

    import torch

    from b200sht.semilag import (CartesianWind, SphericalGridTables, departure_points,
                                 gather_batch, zero_stencil)

    nlev, nlat, nlon = shape
    lat = (np.arange(nlat) + 0.5) * np.pi / nlat - 0.5 * np.pi
    tables = SphericalGridTables.create(types.SimpleNamespace(
        nlat=nlat, nlon=nlon, lat_rad=lat, lon_rad=np.arange(nlon) * 2 * np.pi / nlon,
        radius_m=6371220.0), dtype=torch.float64)
    gen = torch.Generator(device="cuda").manual_seed(3)
    fields = [torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
              for _ in range(3)]
    for got, want in zip(gather_batch(fields, zero_stencil(tables, nlev)), fields):
        assert torch.equal(got, want)
    rest = torch.zeros(shape, dtype=torch.float64, device="cuda")
    st, d = departure_points(CartesianWind(rest, rest, rest, rest), tables, 300.0)
    assert torch.equal(st.level, torch.arange(nlev, dtype=torch.float64, device="cuda")
                       [:, None, None].expand(shape))
    assert float((st.phi - torch.as_tensor(lat, device="cuda")[None, :, None]).abs().max()) < 1e-12
    assert d.displacement_max_levels == 0.0 and d.displacement_max_m < 1e-6


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_block_and_move_array_entries(dtype):
    """The C entries beside the ones the Python calls take: gathers of one
    contiguous block and the band search with move arrays, bit for bit."""
    import torch

    from b200sht import _lib
    from b200sht.semilag import CartesianWind, Stencil, departure_points, gather_batch

    tables, at, field = _setup(getattr(torch, dtype))
    block = torch.stack([field() for _ in range(3)])
    ptr = lambda t: t.data_ptr()  # noqa: E731
    stream = torch.cuda.current_stream().cuda_stream
    nlev = block.shape[1]
    band = tables.window(slice(4, 30), slice(9, 24))
    for window in (None, band):
        pts = [x if window is None else x[:, 9:24].contiguous() for x in at]
        src = block if window is None else block[:, :, 4:30].contiguous()
        want = gather_batch(list(src), Stencil(*pts, tables=tables, window=window))
        got = torch.empty((3, *pts[0].shape), dtype=block.dtype, device="cuda")
        name, handle = (("sht_sl_gather", tables._handle) if window is None
                        else ("sht_sl_gather_band", window._handle))
        _lib.call(name, handle, 4, _lib.SHT_SL_QUASI_MONOTONE, 0, ptr(src), 3, nlev,
                  *[ptr(x) for x in pts], ptr(got), None, stream)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    wind = [30.0 * field()[:, 4:30].contiguous() for _ in range(3)]
    wind.append(1e-3 * field()[:, 4:30].contiguous())
    ahead = [w[:, band.local].contiguous() for w in wind]
    st, d = departure_points(CartesianWind(*wind), tables, 300.0, window=band,
                             extrapolated=CartesianWind(*ahead))
    outs = [torch.empty_like(st.xi) for _ in range(5)]
    _lib.call("sht_sl_departure_band", band._handle, 0, nlev, *[ptr(x) for x in wind + ahead], 3,
              300.0, tables.radius_m, *[ptr(x) for x in outs], stream)
    assert all(torch.equal(a, b) for a, b in zip((st.xi, st.phi, st.level), outs))
    assert d.move_max_m == float(outs[3].max()) and d.move_max_levels == float(outs[4].max())
