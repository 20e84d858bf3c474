"""Coefficient <-> folded-row layout at the edges of its blocks (32 orders, 4
or 2 degrees, 32 columns of planes and fields), against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("T", [30, 31, 32, 34])
def test_blocks_of_orders_and_columns(T, precision):
    from b200sht import SphericalHarmonicTransform, VorticityDivergenceOperator
    from b200sht.synthetic import red_spectrum
    from oracle.dense_sht import DenseSHT

    kw = dict(nlat=T + 4, nlon=2 * T + 4, dealias_factor=1.0)
    t = SphericalHarmonicTransform.create(T, precision=precision, **kw)
    vec = VorticityDivergenceOperator(t)
    ora = DenseSHT(T, **kw)
    np_ = t.backend.to_numpy
    tol = 1e-12 if precision == "float64" else 2e-6
    rel = lambda a, b: float(np.max(np.abs(np_(a) - b)) / np.max(np.abs(b)))  # noqa: E731
    for planes in (5, 15, 16, 17, 32, 33):
        c = red_spectrum(T, planes, T + planes)
        d = red_spectrum(T, planes, T + planes + 1)
        grid = ora.inverse(c)
        u, v = ora.wind_from_vordiv(c, d)
        assert rel(t.inverse(c), grid) < tol
        assert rel(t.forward(grid), ora.forward(grid)) < tol
        for a, b in zip(vec.wind_from_vordiv(c, d), (u, v)):
            assert rel(a, b) < tol
        # 8 T ulps of the O(T)-amplified wind rows
        vtol = tol if precision == "float64" else 8 * T * 6e-8
        got, want = vec.vordiv_from_wind(u, v), ora.vordiv_from_wind(u, v)
        for a, b in zip(got, want):
            assert rel(a, b) < vtol
            assert not np.any(np_(a)[:, 0, 1:]) and not np.any(np_(a)[:, :, 0].imag)
    t.check_device()
