"""The longitude FFTs at row lengths that take each radix of the pass plan
(odd and even lengths, one pass and several, primes with and without a radix
of their own) and at plane counts around a CTA's columns, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nlon / 2 = 6, 7, 9, 10, 11, 13, 15, 16, 17, 2 x 19, 25, 5 x 7, 96, 3 x 125
LONGITUDES = [12, 14, 18, 20, 22, 26, 30, 32, 34, 76, 50, 70, 192, 750]


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("nlon", LONGITUDES)
def test_every_radix_against_the_oracle(nlon, precision):
    from b200sht import SphericalHarmonicTransform, VorticityDivergenceOperator
    from b200sht.synthetic import red_spectrum
    from oracle.dense_sht import DenseSHT

    T = 5 if nlon < 100 else 17
    nlat = T + 4 + nlon % 4 // 2  # odd and even row counts
    kw = dict(nlat=nlat, nlon=nlon, dealias_factor=1.0)
    t = SphericalHarmonicTransform.create(T, precision=precision, **kw)
    ora = DenseSHT(T, **kw)
    np_ = t.backend.to_numpy
    tol = 1e-12 if precision == "float64" else 2e-6
    rel = lambda a, b: float(np.max(np.abs(np_(a) - b)) / np.max(np.abs(b)))  # noqa: E731
    for planes in (1, 2, 7, 9):
        rng = np.random.default_rng(nlon + planes)
        field = rng.standard_normal((planes, nlat, nlon))  # every zonal wavenumber, not only m <= T
        coeff = red_spectrum(T, planes, nlon + planes)
        assert rel(t.fourier_waist(field).values, ora.fourier(field)) < tol
        assert rel(t.inverse(coeff), ora.inverse(coeff)) < tol
        assert rel(t.inverse_zonal_derivative(coeff), ora.inverse_zonal_derivative(coeff)) < tol
        for a, b in zip(t.gradient(coeff), ora.gradient(coeff)):
            assert rel(a, b) < tol
        wind = VorticityDivergenceOperator(t).wind_from_vordiv(coeff, coeff[::-1].copy())
        for a, b in zip(wind, ora.wind_from_vordiv(coeff, coeff[::-1].copy())):
            assert rel(a, b) < tol
    t.check_device()
