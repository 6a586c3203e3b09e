"""Survey correlations at the edges of what they accept, against the oracle: an
observer at the centre of a cell, many short rows."""
import numpy as np
import pytest

import fftcorr_b200 as fb
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
