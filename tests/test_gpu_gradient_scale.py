"""The gradient's scales 1 / a and 1 / (a cos phi) are applied as divisions,
not as reciprocals rounded once, whose error every value of a row would share."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fft", [0, 1])
@pytest.mark.parametrize("planes", [255, 256])
def test_single_precision_gradient_has_no_row_scale_error(fft, planes):
    """The factor that fits each FP32 gradient row to the unscaled derivative
    divided by a cos phi or a.  Where one order carries a row its rounding, up
    to 6e-8 of the value and of either transform, is that of a whole plane:
    below 6e-8 / sqrt(255) = 4e-9 in the mean, three or four times that in the
    worst of 130 rows.  A rounded reciprocal of this radius is 2.6e-8 off, and
    of a row's factor up to 6e-8."""
    import torch

    from b200sht import SphericalHarmonicTransform
    from b200sht.autotune import set_tuning
    from b200sht.synthetic import red_spectrum

    radius = 6371220.0
    t = SphericalHarmonicTransform.create(84, nlat=130, nlon=256, radius_m=radius)
    set_tuning(t, fft=fft)
    c = torch.as_tensor(red_spectrum(84, planes)).to(t.backend.device, torch.complex64)
    cos = torch.as_tensor(t.grid.cos_lat, device=t.backend.device).float()
    east, north = (x.double() for x in t.gradient(c))
    rows = (cos * radius).double()[:, None]  # as the kernel forms it, in FP32
    for got, want in ((east, t.inverse_zonal_derivative(c).double() / rows),
                      (north, t.inverse_meridional_derivative(c).double() / radius)):
        scale = (got * want).sum((0, 2)) / (want * want).sum((0, 2))
        assert float((scale - 1.0).abs().max()) < 1.7e-8
