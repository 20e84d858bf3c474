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


@pytest.mark.parametrize("nlon, T, bound", [(54, 16, 1.018e-7), (486, 30, 1.405e-7)])
def test_radix_three_rounds_its_products_with_their_sums(nlon, T, bound):
    """The FP32 error of transforms by threes, against 64 bits, over 60 planes
    (0.2 % from seed to seed): 0.997e-7 and 1.38e-7 of the spectrum where a
    butterfly's product rounds with the sum it goes into, 1.039e-7 and 1.43e-7
    where it rounds first; the bounds lie between."""
    import torch

    from b200sht import SphericalHarmonicTransform

    t = SphericalHarmonicTransform.create(T, nlat=max(40, (3 * T + 5) // 2), nlon=nlon)
    gen = torch.Generator(device="cuda").manual_seed(1)
    g = torch.randn(60, t.grid.nlat, nlon, generator=gen, device="cuda")
    want = torch.fft.rfft(g.double(), dim=-1)[..., :T + 1] / nlon
    got = t.fourier_waist(g).take().to(torch.complex128)
    assert float((got - want).norm() / want.norm()) < bound
