"""The dose readout of a world of more voxels than a capped grid of 524,280 blocks of 256
threads covers, at two voxels a thread (2^28 - 4096) and at one (half of that): every voxel
is written, and those behind either mark are the plain FP64 formula on the tally."""
import ctypes as C

import numpy as np
import pytest

from opendxmc_gb300 import native as N
from opendxmc_gb300 import phantoms as P

pytestmark = pytest.mark.gpu

DIMS, SPACING = (1024, 1024, 257), (0.05, 0.05, 0.05)
MARKS = (524_280 * 256, 524_280 * 512)


def test_every_voxel_of_a_large_world_is_written(gpu):
    import torch

    n = int(np.prod(DIMS))
    assert n > MARKS[1]
    w = gpu.GpuWorld(DIMS, SPACING, [P.WATER])
    w.set_data(np.full(n, 1.25, np.float32), np.zeros(n, np.uint8))
    w.build()
    beam = P.dx_beam_params(field_cm=40.0, particles=2_000_000, exposures=1)
    hist = w.run(beam, gpu.run_options(seed=4))["n_histories"]
    e, e2, c = w.tally()
    s = 1.602176634e-10 / (SPACING[0] * SPACING[1] * SPACING[2]) / 1.25
    out = [torch.empty(n + 1, dtype=t, device="cuda") for t in (torch.float64, torch.float64, torch.int64)]
    for shift in (0, 1):  # on a 16-byte boundary: two voxels a thread; off it: one
        for x in out:
            x.fill_(-7)
        torch.cuda.synchronize()  # the library reads out on a stream of the world's own
        at = [x.data_ptr() + 8 * shift for x in out]
        N.check(N.lib().dxmcg_world_read_dose(w._h, C.cast(at[0], C.POINTER(C.c_double)),
                                              C.cast(at[1], C.POINTER(C.c_double)),
                                              C.cast(at[2], C.POINTER(C.c_uint64))))
        # one element of each is beside the arrays and stays as it is
        assert [int((x == -7).sum()) for x in out] == [1, 1, 1]
        assert [int(x[0 if shift else n]) for x in out] == [-7, -7, -7]
        for mark in MARKS:
            a, b = mark - 5000, min(n, mark + 1_500_000)
            d, v, k = (x[a + shift:b + shift].cpu().numpy() for x in out)
            assert c[mark:b].sum() > 0
            x = e2[a:b] - e[a:b] * e[a:b] / hist
            np.testing.assert_array_equal(d, e[a:b] * s)
            np.testing.assert_array_equal(v, np.where(x > 0, x, 0.0) * s * s)
            np.testing.assert_array_equal(k, c[a:b].astype(np.int64))
    w.close()
