"""Where a denoised dose map is written changes nothing of it: pageable memory (copied after
the network) and pinned memory (zeroed during the network, the tissue bricks stored by the
last convolution), on grids that take the sparse pass and one that does not."""
import ctypes as C

import numpy as np
import pytest

from opendxmc_gb300 import native as N
from opendxmc_gb300 import phantoms as P

pytestmark = pytest.mark.gpu


def denoise(w, net, out):
    scale = C.c_double(0)
    N.check(N.lib().dxmcg_world_denoise(w._h, net._h, 0.0, out.ctypes.data_as(C.POINTER(C.c_double)), C.byref(scale)))
    return scale.value


@pytest.mark.parametrize("dims", [(128, 128, 80), (104, 72, 136), (32, 32, 32)])
def test_pinned_and_pageable_destinations(gpu, dims):
    torch = pytest.importorskip("torch")
    ph = P.torso_phantom(dims=dims, spacing=(0.3, 0.3, 0.35), seed=2)
    w = gpu.GpuWorld(ph.dims, ph.spacing, ph.materials, 1)
    w.set_data(ph.density, ph.material)
    w.build()
    w.run(P.ct_spiral_params(particles=2000, scan_cm=20.0), gpu.run_options(seed=3))
    net = gpu.Denoiser((16, 32, 64, 128), seed=1)
    n = dims[0] * dims[1] * dims[2]
    pageable = np.full(n, np.nan)
    pinned = torch.full((n + 1,), float("nan"), dtype=torch.float64).pin_memory()
    s1 = denoise(w, net, pageable)
    s2 = denoise(w, net, pinned[1:].numpy())
    assert s1 == pytest.approx(s2, rel=1e-12) and s1 > 0
    got = pinned[1:].numpy()
    assert np.all(np.isfinite(pageable)) and np.isnan(pinned[0].item())
    np.testing.assert_array_equal(got == 0.0, pageable == 0.0)
    # the scale is a sum of FP64 atomics: its last bits move the bf16 input at most by a
    # rounding, 2^-8 of a value, and rarely
    assert np.linalg.norm(got - pageable) <= 2.0 ** -8 * np.linalg.norm(pageable)
