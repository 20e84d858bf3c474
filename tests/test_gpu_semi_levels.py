"""The stage solve at level counts around its row tiles and its shared-memory
limit, and at truncations around its 32-order blocks, on both sides of the
sizes from which its own kernel runs, against the oracle; and fused onto the
synthesis."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision, tol", [("float64", 1e-11), ("float32", 1e-5)])
@pytest.mark.parametrize("T, nlev", [(5, 1), (31, 7), (32, 8), (33, 9), (63, 15), (40, 16),
                                     (21, 47), (21, 48), (21, 75), (21, 80),
                                     # by the kernel of its own
                                     (223, 1), (223, 7), (224, 8), (223, 9), (223, 15), (160, 16),
                                     (170, 40), (170, 41), (96, 50), (96, 66)])
def test_solve_against_the_oracle(T, nlev, precision, tol):
    import torch

    from b200sht import SphericalHarmonicTransform
    from b200sht.semi_implicit import VerticalModeOperator, VerticalModeSemiImplicit
    from b200sht.synthetic import red_spectrum, seeded_vertical_operator
    from oracle.dense_sht import solve_shifted

    if precision == "float64" and nlev > 48:
        pytest.skip("the operators of this many levels do not fit an SM in FP64")
    t = SphericalHarmonicTransform.create(T, precision=precision)
    op = VerticalModeOperator(*seeded_vertical_operator(nlev))
    d, th = 1e-5 * red_spectrum(T, nlev, 1), 20.0 * red_spectrum(T, nlev, 2)
    lp = 0.1 * red_spectrum(T, 1, 3)[0]
    d[:, 0, 0], th[:, 0, 0], lp[0, 0] = 1e-6, 300.0, 11.5  # degree zero passes through
    want = solve_shifted(d, th, lp, op.b_matrix, op.c_matrix, op.eigenvalues, op.eigenvectors, 150.0)
    solver = VerticalModeSemiImplicit()
    got = solver.solve_arrays(t, op, 150.0, d, th, lp)
    for a, b in zip(got, want):
        a = t.backend.to_numpy(a)
        assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(b))
        assert not np.any(np.triu(np.ones(a.shape[-2:], dtype=bool), 1) & (a != 0))
    # in place, and with the synthesis of the solved divergence fused on
    ins = [t._spec_in(x) for x in (d, th, lp)]
    grid = t._empty_grid((nlev,))
    solver.solve_and_synthesize_into(t, op, 150.0, *ins, *ins, grid)
    for a, b in zip(ins, got):
        assert torch.equal(a, b)
    assert torch.equal(grid, t.inverse(got[0]))
    t.check_device()
