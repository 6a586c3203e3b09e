"""Device memory of correlators: an FP32 copy of the density is only held where
FP64 cells are correlated in FP32, and the server's footprint of a correlator
is what it allocates, within a tenth."""
import ctypes

import numpy as np
import pytest

import fftcorr_b200 as fb
from fftcorr_b200 import _lib
from fftcorr_b200.serve import CAT_CLUSTERED_BOX, JobSpec, catalog_spec
from oracle import fc_oracle as O
from test_gpu_parity import FP64_RTOL, _compare_results

pytestmark = pytest.mark.gpu

POSMIN = np.array([-160.0, -160.0, 20.0])


def _device_bytes():
    b = ctypes.c_size_t()
    _lib.call("fc_device_bytes", ctypes.byref(b))
    return b.value


@pytest.mark.parametrize("kind", ["periodic", "survey"])
def test_density_copy_on_first_fp64_cells(kind):
    shape, cell = (64, 60, 64), 10.0
    values = np.random.default_rng(3).standard_normal(shape).astype(np.float32)
    if kind == "periodic":
        args = (cell, 0, 100.0, 10.0, 0.2, 0.02, 2)
        c, oracle = fb.PeriodicCorrelator(shape, *args, precision="fp32"), O.periodic_correlate
    else:
        args = (cell, POSMIN, 2, 100.0, 10.0, 0.2, 0.02, 2)
        c, oracle = fb.Correlator(shape, *args, precision="fp32"), O.survey_correlate
    ref = oracle(values.astype(np.float64), *args)
    grids = {}
    for precision in ("fp32", "fp64"):
        g = fb.ConfigSpaceGrid.from_geometry(shape, POSMIN, cell, precision=precision)
        _lib.call("fc_grid_upload", g.handle, _lib.dptr(values.astype(np.float64)))
        grids[precision] = g
    before = _device_bytes()
    c.autocorrelate(grids["fp32"])
    assert _device_bytes() == before
    _compare_results(c.results(), ref, FP64_RTOL, "FP32 cells", fp32=True)
    _lib.call("fc_fault_inject", _lib.FC_FAULT_DEVICE_ALLOC, 1)
    with pytest.raises(MemoryError):
        c.autocorrelate(grids["fp64"])
    assert _device_bytes() == before
    for _ in range(2):
        c.autocorrelate(grids["fp64"])
        assert _device_bytes() == before + 4 * values.size
        _compare_results(c.results(), ref, FP64_RTOL, "FP64 cells", fp32=True)


@pytest.mark.parametrize("kind", ["periodic", "survey"])
@pytest.mark.parametrize("n2", [128, 120, 105])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_footprint_of_a_correlator(kind, n2, precision):
    """The bytes by which larger subgrids make a correlator grow, from the
    server's estimate and from what is allocated: the estimate holds them, and
    is at most a quarter above (cells in range are counted by volume)."""
    shape, cell = (128, 96, n2), 10.0
    data = catalog_spec(CAT_CLUSTERED_BOX, n=1000, boxsize=900.0, ncentres=10, sigma=5.0,
                        seed=1)

    def both(rmax, kmax):
        job = JobSpec(kind, shape, cell, data, data if kind == "survey" else None,
                      posmin=POSMIN, rmax=rmax, dr=rmax / 8, kmax=kmax, dk=kmax / 8,
                      maxell=2, precision=precision)
        args = (0, rmax, rmax / 8, kmax, kmax / 8, 2)
        before = _device_bytes()
        if kind == "periodic":
            c = fb.PeriodicCorrelator(shape, cell, *args, precision=precision)
        else:
            c = fb.Correlator(shape, cell, POSMIN, *args, precision=precision)
        made = _device_bytes() - before
        del c
        return job.footprint, made

    estimate, made = np.subtract(both(397.0, 0.3), both(53.0, 0.05))
    assert made <= estimate <= 1.25 * made, (estimate, made)
