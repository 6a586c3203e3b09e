"""Catalogs of more than 40 particles per scatter unit (2 x 8 x 8 cells) on
average take the scatter's dense form, CIC's another kernel: the counts at that
line, and many more, units of no, one and thousands of particles among them,
against the oracle."""
import numpy as np
import pytest

import fftcorr_b200 as fb
from oracle import fc_oracle as O
from test_scatter_units import _unit_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", [0, 1, 3])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [3840, 3841, 14000])   # 96 units
def test_dense_form(scheme, precision, n):
    shape = (16, 24, 32)
    posw = _unit_points(np.random.default_rng(5), shape,
                        [1, 31, 200, n - 3232, 1000, 2000])
    assert len(posw) == n
    ref, _ = O.mass_assign(posw, shape, [0.0] * 3, 1.0, scheme, True)
    grid = fb.ConfigSpaceGrid.from_geometry(shape, [0.0] * 3, 1.0, precision=precision)
    fb.MassAssignor(grid, scheme, True, 0).add_particles(posw)
    # FP64 sums in another order; an FP32 cell rounds once per unit that
    # reaches it (at most 8), 6e-8 of its value each.
    tol = 1e-12 if precision == "fp64" else 8 * 6e-8
    assert np.max(np.abs(np.asarray(grid) - ref)) <= tol * np.max(np.abs(ref))
