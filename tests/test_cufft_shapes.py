"""What runs through cuFFT, sides with a prime factor above 7 and long rows: the batched form
beside fused boxes, and an FFT plan that cannot be made (raised on the host
before the cuFFT call)."""
import ctypes

import numpy as np
import pytest

from conftest import clustered_catalog
from oracle import fc_oracle as O

import fftcorr_b200 as fb
from fftcorr_b200 import _lib
from fftcorr_b200.batch import PeriodicBatch
from test_batch import _batch, _single_box
from test_gpu_parity import FP64_RTOL, _compare_results

pytestmark = pytest.mark.gpu

POSMIN = np.array([-160.0, -160.0, 20.0])


@pytest.fixture(autouse=True)
def _disarm():
    yield
    _lib.call("fc_fault_inject", _lib.FC_FAULT_FFT_PLAN, 0)


def _device_bytes():
    b = ctypes.c_size_t()
    _lib.call("fc_device_bytes", ctypes.byref(b))
    return b.value


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_batch_equals_single_box_path(precision):
    boxes = []
    for shape, n, seed in [((22, 22, 22), 20000, 1), ((33, 26, 39), 30000, 2),
                           ((32, 32, 32), 30000, 3), ((26, 44, 22), 4000, 4)]:
        posw = clustered_catalog(n, [0, 0, 0], 10.0 * np.array(shape), seed, ncenters=30)
        boxes.append((shape, 10.0, posw))
    b = _batch(boxes, precision)
    b.run()
    for i, (shape, cell, posw) in enumerate(boxes):
        ref, _ = _single_box(shape, cell, posw, precision)
        got = b.results(i)
        for key in ("rcounts", "kcounts", "rhist", "khist"):
            np.testing.assert_array_equal(got[key], ref[key], err_msg=f"box {i} {key}")
        assert got["zerolag"] == ref["zerolag"]


@pytest.mark.parametrize("kind", ["periodic", "survey"])
def test_plan_failure_leaves_nothing_behind(kind):
    shape, cell = (22, 26, 33), 10.0
    if kind == "periodic":
        args = (cell, 0, 60.0, 7.0, 0.25, 0.02, 2)
        make, oracle = fb.PeriodicCorrelator, O.periodic_correlate
    else:
        args = (cell, POSMIN, 2, 60.0, 10.0, 0.2, 0.04, 2)
        make, oracle = fb.Correlator, O.survey_correlate
    before = _device_bytes()
    _lib.call("fc_fault_inject", _lib.FC_FAULT_FFT_PLAN, 1)
    with pytest.raises(_lib.FcError) as e:
        make(shape, *args)
    assert e.value.code == _lib.FC_ERR_CUFFT
    assert _device_bytes() == before
    grid = np.random.default_rng(5).standard_normal(shape)
    c = make(shape, *args)
    c.autocorrelate(grid)
    _compare_results(c.results(), oracle(grid, *args), FP64_RTOL, kind)


LARGE = (242, 264, 286)   # a k-subgrid of 18M cells, 150 MB in FP64


@pytest.mark.parametrize("kind", ["periodic", "survey"])
def test_large_subgrids_take_turns(kind):
    """A k-subgrid that reaches the Nyquist frequency is larger than the grid:
    at ell <= 4 the multipoles use one pair of subgrids in turn, and their
    histograms are reduced one by one, which gives the bits of ell <= 2 (a pair
    each) and holds less."""
    grid = np.random.default_rng(6).standard_normal(LARGE)

    def run(maxell):
        args = (60.0, 7.0, 0.35, 0.03, maxell)
        before = _device_bytes()
        if kind == "periodic":
            c = fb.PeriodicCorrelator(LARGE, 10.0, 0, *args, precision="fp32")
        else:
            c = fb.Correlator(LARGE, 10.0, POSMIN, 2, *args, precision="fp32")
        made = _device_bytes() - before
        c.autocorrelate(grid)
        first = c.results()
        c.autocorrelate(grid)
        for key in ("rhist", "khist"):
            np.testing.assert_array_equal(first[key], c.results()[key])
        return made, first

    made2, two = run(2)
    made4, four = run(4)
    assert made4 < made2
    for key in ("rhist", "khist", "rcounts", "kcounts"):
        np.testing.assert_array_equal(four[key][:2], two[key])
        assert np.all(np.isfinite(four[key])) and np.any(four[key][2] != 0)
    assert four["zerolag"] == two["zerolag"]


def test_batch_with_large_subgrids():
    """A batch reduces all histograms at its end, from a pair of subgrids each."""
    posw = clustered_catalog(20000, [0, 0, 0], 10.0 * np.array(LARGE), 1, ncenters=30)
    args = (60.0, 7.0, 0.35, 0.03, 4)
    b = PeriodicBatch([(LARGE, 10.0, posw)], fb.DistributionScheme.CLOUD_IN_CELL, *args, 0,
                      "fp32", tune=False)
    b.run()
    g = fb.ConfigSpaceGrid.from_geometry(LARGE, [0, 0, 0], 10.0, precision="fp32")
    ma = fb.MassAssignor(g, fb.DistributionScheme.CLOUD_IN_CELL, True, 0)
    ma.add_particles(posw)
    mean = ma.totw / float(np.prod(LARGE))
    g -= mean
    g *= 1.0 / mean
    c = fb.PeriodicCorrelator(LARGE, 10.0, 0, *args, precision="fp32")
    c.autocorrelate(g)
    for key in ("rcounts", "kcounts", "rhist", "khist"):
        np.testing.assert_array_equal(b.results(0)[key], c.results()[key])


def test_fused_surveys_make_no_plan_that_could_fail():
    args = (10.0, POSMIN, 2, 60.0, 10.0, 0.2, 0.04, 2)
    _lib.call("fc_fault_inject", _lib.FC_FAULT_FFT_PLAN, 1)
    fb.Correlator((32, 30, 36), *args)
    with pytest.raises(_lib.FcError):   # the planned failure is still to come
        fb.Correlator((22, 26, 33), *args)


@pytest.mark.parametrize("shape", [(4, 6, 4096), (5, 4, 2592), (2, 3, 2625)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_long_rows(shape, precision, monkeypatch):
    """Rows of more than 2560 cells: cuFFT's path by itself and when asked for
    give the same bits; those of 2560 run through the fused passes."""
    grid = np.random.default_rng(9).standard_normal(shape)
    args = (10.0, POSMIN, 2, 10.0 * min(shape), 4.0, 0.1, 0.02, 4)
    c = fb.Correlator(shape, *args, precision=precision)
    c.autocorrelate(grid)
    got = c.results()
    monkeypatch.setenv("FFTCORR_B200_FFT", "cufft")
    c = fb.Correlator(shape, *args, precision=precision)
    c.autocorrelate(grid)
    for key in ("rcounts", "kcounts", "rhist", "khist"):
        np.testing.assert_array_equal(got[key], c.results()[key])
    _compare_results(got, O.survey_correlate(grid, *args), FP64_RTOL, "long rows",
                     fp32=precision == "fp32")


@pytest.mark.parametrize("n2", [2048, 2500, 2560, 2401])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_longest_fused_rows(n2, precision):
    shape = (4, 6, n2)
    grid = np.random.default_rng(9).standard_normal(shape)
    args = (10.0, POSMIN, 2, 40.0, 4.0, 0.1, 0.02, 4)
    c = fb.Correlator(shape, *args, precision=precision)
    c.autocorrelate(grid)
    _compare_results(c.results(), O.survey_correlate(grid, *args), FP64_RTOL, "long rows",
                     fp32=precision == "fp32")
