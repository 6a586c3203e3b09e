"""Survey correlations at the edges of what they accept, against the oracle: an
observer at the centre of a cell, many short rows, odd rows of either cell type,
separations that are not their mirror images to the last bit."""
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


@pytest.mark.parametrize("cross", [False, True])
def test_odd_fp32_rows_of_periodic_grids(cross):
    """The same of periodic correlations, which weight no cells."""
    shape = (30, 64, 27)
    rng = np.random.default_rng(13)
    args = (CELL, TSC_ALIASED_CORRECTION, 50.0, 6.0, 0.15, 0.03, 4)
    values = [rng.standard_normal(shape).astype(np.float32) for _ in range(2)]
    results = []
    for precision in ("fp32", "fp64"):
        grids = []
        for v in values:
            g = fb.ConfigSpaceGrid.from_geometry(shape, np.zeros(3), CELL,
                                                 precision=precision)
            _lib.call("fc_grid_upload", g.handle, _lib.dptr(v.astype(np.float64)))
            grids.append(g)
        c = fb.PeriodicCorrelator(shape, *args, precision="fp32")
        if cross:
            c.cross_correlate(*grids)
        else:
            c.autocorrelate(grids[0])
        results.append(c.results())
    ref = O.periodic_correlate(values[0].astype(np.float64), *args,
                               grid2=values[1].astype(np.float64) if cross else None)
    _compare_results(results[0], ref, FP64_RTOL, "odd rows", fp32=True)
    for key in ("rhist", "khist"):
        np.testing.assert_array_equal(results[0][key], results[1][key])


def test_axes_that_are_not_their_own_mirror_image():
    """cell = 17.1 rounds the r axis differently at r and -r (1e-14 of a cell),
    which has to cancel between the two in the sums of a bin.  The field is
    smooth, so that xi is nearly the same in all cells of the small bins and
    their quadrupole cancels but for that.  What the sums would be off by if a
    cell's weight stood for its mirror image is known from the axis: the error
    against the oracle contains it once then, and not at all otherwise."""
    n, cell, r = 64, 17.1, 60
    dr = 24.77   # no cell at the edge of a bin, so the bins of r and -r agree
    axis = -(cell * r) + np.arange(2 * r + 1) * cell
    x = (np.arange(n) - n / 2) / 15.0
    g = np.exp(-0.5 * x * x)
    grid = g[:, None, None] * g[None, :, None] * g[None, None, :]
    posmin = np.array([20000.0, -cell * n / 2, -cell * n / 2])   # along x, far away
    args = (cell, posmin, TSC_ALIASED_CORRECTION, cell * r, dr, 0.1, 0.02, 2)
    c = fb.Correlator((n, n, n), *args)
    c.autocorrelate(grid)
    res, ref = c.results(), O.survey_correlate(grid, *args)
    np.testing.assert_array_equal(res["rcounts"], ref["rcounts"])
    error = ((res["rhist"][1] - ref["rhist"][1]) / ref["rhist"][0])[:10]

    a = axis[r - 16:r + 17]
    xx, yy, zz = np.meshgrid(a, a, a, indexing="ij")
    rr = np.sqrt(xx * xx + yy * yy + zz * zz)
    quadrupole = 2.5 * (3.0 * xx * xx / (rr * rr + 1e-20) - 1.0)
    mirrored = quadrupole.copy()
    mirrored[:16] = quadrupole[::-1, ::-1, ::-1][:16]
    bins = np.floor(rr / dr).astype(int)
    xi = np.exp(-(rr / cell / 15.0) ** 2 / 4.0)
    off = np.array([np.sum(((mirrored - quadrupole) * xi)[bins == b]) / np.sum(xi[bins == b])
                    for b in range(10)])
    share = np.dot(error, off) / np.dot(off, off)
    assert abs(share) < 0.5, (share, error, off)
