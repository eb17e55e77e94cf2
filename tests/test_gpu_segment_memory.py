"""CT segmentation of host arrays that share memory (the outputs of every voxel come from its
own CT number as it was before the call), or that lie off their element's boundary (records
of a file read as they are), against the same FP64 operations in numpy (exact).  The CT
numbers are no integers, so that their last bits count; the largest array is more than one
pass of the kernel's grid."""
import ctypes as C

import numpy as np
import pytest

from opendxmc_gb300 import native as N
from test_gpu_segment_blocks import expected

pytestmark = pytest.mark.gpu


def segment(t, hu, mat, den):
    N.check(N.lib().dxmcg_ct_segment(C.byref(t), hu.ctypes.data_as(C.POINTER(C.c_double)), hu.size,
                                     mat.ctypes.data_as(C.POINTER(C.c_uint8)),
                                     den.ctypes.data_as(C.POINTER(C.c_double))))


def ct_numbers(n):
    return np.random.default_rng(n).uniform(-1100.0, 3200.0, n)


@pytest.mark.parametrize("n", [1, 700, 300_001, 2_500_003])
def test_in_place(gpu, n):
    t = gpu.ct_segmentation_table()
    hu = ct_numbers(n)
    m, d = expected(t, hu)
    mat = np.full(n, 250, dtype=np.uint8)
    segment(t, hu, mat, hu)  # the densities in place of the CT numbers
    np.testing.assert_array_equal(mat, m)
    np.testing.assert_array_equal(hu, d)


@pytest.mark.parametrize("n", [700, 300_001])
def test_materials_over_ct_numbers(gpu, n):
    t = gpu.ct_segmentation_table()
    hu = ct_numbers(n)
    m, d = expected(t, hu)
    mat = hu.view(np.uint8)[5 * n:6 * n]
    den = np.full(n, -3.0)
    segment(t, hu, mat, den)
    np.testing.assert_array_equal(mat, m)
    np.testing.assert_array_equal(den, d)


def off_boundary(n, dtype, shift):
    """n elements that start `shift` bytes behind an element's boundary."""
    size = np.dtype(dtype).itemsize
    return np.zeros(n * size + 2 * size, np.uint8)[shift:shift + n * size].view(dtype)


@pytest.mark.parametrize("hu_shift,den_shift", [(4, 0), (0, 4), (1, 3), (8, 4)])
@pytest.mark.parametrize("n", [1, 129, 600_001])
def test_off_the_element_boundary(gpu, n, hu_shift, den_shift):
    t = gpu.ct_segmentation_table()
    hu, den = off_boundary(n, np.float64, hu_shift), off_boundary(n, np.float64, den_shift)
    assert hu.ctypes.data % 8 == hu_shift % 8 and den.ctypes.data % 8 == den_shift % 8
    hu[:] = ct_numbers(n)
    m, d = expected(t, hu.copy())
    mat = np.full(n, 250, dtype=np.uint8)
    segment(t, hu, mat, den)
    np.testing.assert_array_equal(mat, m)
    np.testing.assert_array_equal(den, d)
