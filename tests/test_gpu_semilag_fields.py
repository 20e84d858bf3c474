"""Gathers of several separate fields (interleaved in groups of 16 bytes, the
rest in a pair and a single) against the one-field call."""
from __future__ import annotations

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

