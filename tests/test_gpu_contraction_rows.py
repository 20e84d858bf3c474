"""FP32 and FP64 contractions at the row counts where the kernel or its row
blocks change: every output is one chain of multiply-adds in the same order,
so a plane's result is the same bits whatever batch it is transformed in."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("T, nlat, nlon", [(9, 15, 30), (48, 74, 150), (62, 95, 192), (90, 137, 288),
                                           (200, 302, 640), (341, 514, 1026)])
def test_a_plane_has_the_same_bits_in_every_batch(T, nlat, nlon, precision):
    import torch

    from b200sht import SphericalHarmonicTransform, VorticityDivergenceOperator
    from b200sht.synthetic import red_spectrum

    t = SphericalHarmonicTransform.create(T, nlat=nlat, nlon=nlon, precision=precision)
    vec = VorticityDivergenceOperator(t)
    coeff = torch.as_tensor(red_spectrum(T, 37, 5), device=t.backend.device).to(t.backend.complex_dtype)
    grid = t.inverse(coeff)
    spec = t.forward(grid)
    east, north = t.gradient(coeff)
    u, v = vec.wind_from_vordiv(coeff, spec)
    zeta, div = vec.vordiv_from_wind(u, v)
    # rows: 2 per padded plane (8 and below take the streaming kernel), 4 per
    # plane of a vector call; blocks of 64 (FP32) or 32 (FP64) rows and halves
    for planes in (1, 2, 4, 5, 8, 15, 16, 17, 31, 33):
        c, s = coeff[:planes].contiguous(), spec[:planes].contiguous()
        assert torch.equal(t.inverse(c), grid[:planes])
        assert torch.equal(t.forward(grid[:planes].contiguous()), s)
        for a, b in zip(t.gradient(c), (east, north)):
            assert torch.equal(a, b[:planes])
        for a, b in zip(vec.wind_from_vordiv(c, s), (u, v)):
            assert torch.equal(a, b[:planes])
        uu, vv = u[:planes].contiguous(), v[:planes].contiguous()
        for a, b in zip(vec.vordiv_from_wind(uu, vv), (zeta, div)):
            assert torch.equal(a, b[:planes])
