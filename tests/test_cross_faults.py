"""A periodic cross correlation whose bins differ under inversion makes passes of
its own with its second grid: every allocation of that failing in turn (raised
on the host before the CUDA call), the correlator stays usable."""
import ctypes

import numpy as np
import pytest

import fftcorr_b200 as fb
from fftcorr_b200 import _lib
from fftcorr_b200.correlate import TSC_ALIASED_CORRECTION
from oracle import fc_oracle as O
from test_gpu_parity import FP64_RTOL, _compare_results

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _disarm():
    yield
    _lib.call("fc_fault_inject", _lib.FC_FAULT_DEVICE_ALLOC, 0)


def _device_bytes():
    b = ctypes.c_size_t()
    _lib.call("fc_device_bytes", ctypes.byref(b))
    return b.value


def test_allocation_failures_in_the_second_grid():
    shape, cell, dr = (36, 32, 40), 2.6, 7.8
    args = (cell, TSC_ALIASED_CORRECTION, cell * 12, dr, 0.3, 0.05, 4)
    rng = np.random.default_rng(8)
    a, b = rng.standard_normal(shape), rng.standard_normal(shape)
    auto = O.periodic_correlate(a, *args)
    c = fb.PeriodicCorrelator(shape, *args)
    c.autocorrelate(a)
    before = _device_bytes()
    for nth in range(1, 40):
        _lib.call("fc_fault_inject", _lib.FC_FAULT_DEVICE_ALLOC, nth)
        try:
            c.cross_correlate(a, b)
        except MemoryError:
            assert _device_bytes() == before, f"allocation {nth}"
            c.autocorrelate(a)
            _compare_results(c.results(), auto, FP64_RTOL, f"after allocation {nth}")
            continue
        break
    assert nth > 5
    cross = O.periodic_correlate(a, *args, grid2=b)
    _compare_results(c.results(), cross, FP64_RTOL, "cross")
    c.autocorrelate(a)
    _compare_results(c.results(), auto, FP64_RTOL, "auto")
    c.cross_correlate(a, b)
    _compare_results(c.results(), cross, FP64_RTOL, "cross again")
