"""The split-FP16 contraction where its K steps are few, odd or many (one to
several per accumulator segment) and its row blocks partial, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [3, 15, 33, 64, 97, 130])
def test_split_against_the_oracle(T):
    from b200sht import SphericalHarmonicTransform
    from b200sht.synthetic import red_spectrum
    from oracle.dense_sht import DenseSHT

    kw = dict(nlat=T + 6, nlon=2 * T + 6, dealias_factor=1.0)
    t = SphericalHarmonicTransform.create(T, precision="split16", **kw)
    ora = DenseSHT(T, **kw)
    np_ = t.backend.to_numpy
    norm = lambda a, b: float(np.linalg.norm((np_(a) - b).ravel()) / np.linalg.norm(b.ravel()))  # noqa: E731
    for planes in (1, 33, 65):
        c = red_spectrum(T, planes, T + planes)
        grid = ora.inverse(c)
        # 22-bit operands and truncated sums: 2e-6 relative L2 is the path's bound
        assert norm(t.inverse(c), grid) < 2e-6
        assert norm(t.forward(grid), ora.forward(grid)) < 2e-6
        for a, b in zip(t.gradient(c), ora.gradient(c)):
            assert norm(a, b) < 2e-6
    t.check_device()
