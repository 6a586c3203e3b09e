"""The fused passes along axes of every kind of length against the oracle:
single-radix and length-1 axes, odd rows, axes long enough for the narrow
column tiles, and a k-subgrid that reaches the Nyquist planes of even and odd
sides."""
import numpy as np
import pytest

import fftcorr_b200 as fb
from fftcorr_b200.correlate import TSC_ALIASED_CORRECTION
from oracle import fc_oracle as O
from test_gpu_parity import FP64_RTOL, _compare_results

pytestmark = pytest.mark.gpu

CELL = 10.0


@pytest.mark.parametrize("shape", [(7, 450, 9), (486, 5, 14), (12, 432, 250), (1, 30, 21),
                                   (10, 27, 35), (128, 6, 63), (45, 64, 128)])
@pytest.mark.parametrize("kmax", [0.15, 0.35])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_survey_axis_lengths(shape, kmax, precision):
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal(shape), rng.standard_normal(shape)
    posmin = np.array([-40.0, 25.0, -35.0])
    rmax = CELL * min(5, min(shape))
    args = (CELL, posmin, TSC_ALIASED_CORRECTION, rmax, 6.0, kmax, 0.03, 4)
    c = fb.Correlator(shape, *args, precision=precision)
    c.autocorrelate(a)
    _compare_results(c.results(), O.survey_correlate(a, *args), FP64_RTOL, "auto",
                     fp32=precision == "fp32")
    c.cross_correlate(a, b)
    _compare_results(c.results(), O.survey_correlate(a, *args, grid2=b), FP64_RTOL,
                     "cross", fp32=precision == "fp32")


@pytest.mark.parametrize("shape", [(7, 450, 9), (486, 5, 14), (1, 30, 21), (64, 64, 64),
                                   (128, 64, 35), (11, 16, 20)])
@pytest.mark.parametrize("kmax", [0.15, 0.35])
@pytest.mark.parametrize("cell,dr", [(10.0, 6.0), (2.6, 5.2)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_periodic_axis_lengths(shape, kmax, cell, dr, precision):
    """Periodic correlations through the fused passes (11 cells: cuFFT), with
    bins that are the same under inversion (10, 6) and that are not (2.6,
    5.2), where a cross correlation takes the general inverse."""
    rng = np.random.default_rng(7)
    a, b = rng.standard_normal(shape), rng.standard_normal(shape)
    rmax = cell * min(9, min(shape))
    args = (cell, TSC_ALIASED_CORRECTION, rmax, dr, kmax, 0.03, 4)
    fp32 = precision == "fp32"
    if rmax < dr and fp32:
        pytest.skip("no separation bin to take an rms over")
    c = fb.PeriodicCorrelator(shape, *args, precision=precision)
    ref = O.periodic_correlate(a, *args)
    c.autocorrelate(a)
    _compare_results(c.results(), ref, FP64_RTOL, "auto", fp32=fp32)
    c.cross_correlate(a, b)
    _compare_results(c.results(), O.periodic_correlate(a, *args, grid2=b), FP64_RTOL,
                     "cross", fp32=fp32)
    c.autocorrelate(a)
    _compare_results(c.results(), ref, FP64_RTOL, "auto again", fp32=fp32)


@pytest.mark.parametrize("shape", [(64, 64, 64), (40, 64, 66)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_bins_that_differ_under_inversion(shape, precision):
    """cell = 2.6 and dr = 7.8 put cells on bin edges whose rounded mirror
    images lie on the other side, so the inverse may not drop the odd part of
    the correlation: the counts of r and -r differ and every bin matches."""
    cell, dr = 2.6, 7.8
    r = -cell * 12 + np.arange(25) * cell
    d = np.sqrt(r[:, None, None] ** 2 + r[None, :, None] ** 2 + r[None, None, :] ** 2)
    bins = np.floor(d / dr)
    assert np.any(bins != bins[::-1, ::-1, ::-1])
    posmin = np.array([-30.0, 25.0, -35.0])
    a = np.random.default_rng(6).standard_normal(shape)
    args = (cell, posmin, TSC_ALIASED_CORRECTION, cell * 12, dr, 0.3, 0.05, 4)
    c = fb.Correlator(shape, *args, precision=precision)
    c.autocorrelate(a)
    _compare_results(c.results(), O.survey_correlate(a, *args), FP64_RTOL, "auto",
                     fp32=precision == "fp32")
