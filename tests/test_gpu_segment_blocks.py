"""CT segmentation of host arrays at the edges of its blocks, of a warp's run of 128 voxels and
of the vector accesses' alignment, against the same FP64 operations in numpy (exact)."""
import ctypes as C

import numpy as np
import pytest

from opendxmc_gb300 import native as N

pytestmark = pytest.mark.gpu

BLOCK = 1 << 19


def expected(t, hu):
    n_sep = t.n_materials - 1
    m = np.searchsorted(np.array(t.separator[:n_sep]), hu, side="right").astype(np.uint8)
    w, a = t.water_attenuation * t.water_density, t.air_attenuation * t.air_density
    return m, np.maximum(((w - a) * hu / 1000.0 + w) / np.array(t.attenuation[:n_sep + 1])[m], 0.0)


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1000, BLOCK - 1, BLOCK, BLOCK + 130, 3 * BLOCK + 77])
@pytest.mark.parametrize("offset", [0, 1])
def test_blocks_and_runs(gpu, n, offset):
    t = gpu.ct_segmentation_table()
    rng = np.random.default_rng(n + offset)
    hu = np.empty(n + offset)[offset:]
    hu[:] = np.rint(rng.uniform(-1100.0, 3200.0, n))
    hu[::7] += 0.25  # no integer: computed, not looked up
    mat = np.full(n + offset + 1, 250, dtype=np.uint8)  # one element beyond stays as it is
    den = np.full(n + offset + 1, -3.0)
    N.check(N.lib().dxmcg_ct_segment(C.byref(t), hu.ctypes.data_as(C.POINTER(C.c_double)), n,
                                     mat[offset:].ctypes.data_as(C.POINTER(C.c_uint8)),
                                     den[offset:].ctypes.data_as(C.POINTER(C.c_double))))
    m, d = expected(t, hu)
    np.testing.assert_array_equal(mat[offset:offset + n], m)
    np.testing.assert_array_equal(den[offset:offset + n], d)
    assert mat[-1] == 250 and den[-1] == -3.0 and (mat[:offset] == 250).all() and (den[:offset] == -3.0).all()
