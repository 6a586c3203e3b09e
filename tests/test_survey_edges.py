"""Survey correlations at the edges of what they accept, against the oracle: an
observer at the centre of a cell, many short rows, odd rows of either cell type."""
import numpy as np
import pytest

import fftcorr_b200 as fb
from fftcorr_b200 import _lib
from fftcorr_b200.correlate import TSC_ALIASED_CORRECTION
from oracle import fc_oracle as O
from test_gpu_parity import FP64_RTOL, _compare_results

pytestmark = pytest.mark.gpu

CELL = 10.0


def _survey(shape, posmin, precision, label):
    grid = np.random.default_rng(11).standard_normal(shape)
    args = (CELL, posmin, TSC_ALIASED_CORRECTION, CELL * min(5, min(shape)), 6.0, 0.15,
            0.03, 4)
    c = fb.Correlator(shape, *args, precision=precision)
    c.autocorrelate(grid)
    _compare_results(c.results(), O.survey_correlate(grid, *args), FP64_RTOL, label,
                     fp32=precision == "fp32")


# Odd rows, mixed-radix even rows, power-of-two rows.
@pytest.mark.parametrize("n", [15, 27, 30, 64])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_observer_at_the_centre_of_a_cell(n, precision):
    """1 / r^4 overflows FP32 in that cell, whose weight is 0."""
    posmin = np.full(3, -CELL * (n // 2 + 0.5))
    _survey((n, n, n), posmin, precision, f"observer in cell {n // 2}")


# Rows of which a CTA of the z pass takes more than it has threads (on 148 SMs
# from about 10700 rows).
@pytest.mark.parametrize("shape", [(128, 128, 4), (108, 108, 6), (128, 128, 5),
                                   (128, 128, 7), (120, 90, 9)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_many_short_rows(shape, precision):
    _survey(shape, np.array([-400.0, 250.0, -30.0]), precision, "short rows")


@pytest.mark.parametrize("shape", [(30, 28, 27), (64, 32, 45)])
@pytest.mark.parametrize("cross", [False, True])
def test_odd_fp32_rows_take_either_cell_type(shape, cross):
    """Odd rows of FP32 correlations weight FP32 and FP64 cells in FP64: the
    same values in either type give the same bits."""
    rng = np.random.default_rng(12)
    posmin = np.array([-40.0, 25.0, -35.0])
    args = (CELL, posmin, TSC_ALIASED_CORRECTION, 50.0, 6.0, 0.15, 0.03, 4)
    values = [rng.standard_normal(shape).astype(np.float32) for _ in range(2)]
    results = []
    for precision in ("fp32", "fp64"):
        grids = []
        for v in values:
            g = fb.ConfigSpaceGrid.from_geometry(shape, posmin, CELL, precision=precision)
            _lib.call("fc_grid_upload", g.handle, _lib.dptr(v.astype(np.float64)))
            grids.append(g)
        c = fb.Correlator(shape, *args, precision="fp32")
        if cross:
            c.cross_correlate(*grids)
        else:
            c.autocorrelate(grids[0])
        results.append(c.results())
    ref = O.survey_correlate(values[0].astype(np.float64), *args,
                             grid2=values[1].astype(np.float64) if cross else None)
    _compare_results(results[0], ref, FP64_RTOL, "odd rows", fp32=True)
    for key in ("rhist", "khist"):
        np.testing.assert_array_equal(results[0][key], results[1][key])
