"""The two scatter kernels meet at 32 particles a unit (2 x 8 x 8 cells): unit
counts around it, beside one another in one flush, against the oracle, into
both cell types, with wrapped footprints and with a catalog that is only 8-byte
aligned."""
import ctypes

import numpy as np
import pytest

import fftcorr_b200 as fb
from fftcorr_b200 import _lib
from fftcorr_b200.catalog.device import DeviceCatalog
from oracle import fc_oracle as O

pytestmark = pytest.mark.gpu


def _unit_points(rng, shape, counts):
    """counts[i] points in unit i, i running over the units along x first."""
    nu = [shape[0] // 2, shape[1] // 8, shape[2] // 8]
    out = []
    for i, n in enumerate(counts):
        u = np.array(np.unravel_index(i * 7 % (nu[0] * nu[1] * nu[2]), nu))
        p = np.empty((n, 4))
        p[:, :3] = (u + rng.random((n, 3))) * [2, 8, 8]
        p[:, 3] = rng.uniform(0.5, 1.5, n)
        out.append(p)
    p = np.concatenate(out)
    return p[rng.permutation(len(p))]


@pytest.mark.parametrize("scheme", [0, 1, 3])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shift", [0, 8])
def test_units_around_one_warp(scheme, periodic, precision, shift):
    shape = (16, 24, 32)
    posw = _unit_points(np.random.default_rng(3), shape,
                        [1, 31, 32, 33, 0, 64, 65, 200, 2, 1000, 30, 34])
    n = len(posw)
    ref, _ = O.mass_assign(posw, shape, [0.0] * 3, 1.0, scheme, periodic)
    grid = fb.ConfigSpaceGrid.from_geometry(shape, [0.0] * 3, 1.0, precision=precision)
    ma = fb.MassAssignor(grid, scheme, periodic, 0)
    cat = DeviceCatalog(n + 1)
    _lib.call("fc_memcpy_htod", ctypes.c_void_p(cat.ptr + shift),
              posw.ctypes.data_as(ctypes.c_void_p), posw.nbytes)
    ma.add_particles_device(cat.ptr + shift, n)
    # FP64 sums in another order; an FP32 cell rounds once per unit that
    # reaches it (at most 12), 6e-8 of its value each.
    tol = 1e-12 if precision == "fp64" else 12 * 6e-8
    assert np.max(np.abs(np.asarray(grid) - ref)) <= tol * np.max(np.abs(ref))
    assert ma.num_added == n


def test_dense_catalog_leaves_the_warps_out():
    """More than 40 particles per unit on average: every unit, the nearly empty
    ones too, goes to a CTA."""
    shape = (16, 24, 32)
    posw = _unit_points(np.random.default_rng(4), shape, [4000, 1, 31, 32, 33, 200])
    ref, _ = O.mass_assign(posw, shape, [0.0] * 3, 1.0, 1, True)
    grid = fb.ConfigSpaceGrid.from_geometry(shape, [0.0] * 3, 1.0)
    fb.MassAssignor(grid, 1, True, 0).add_particles(posw)
    assert np.max(np.abs(np.asarray(grid) - ref)) <= 1e-12 * np.max(np.abs(ref))
