"""The dose readout against its plain FP64 formula on the tally it reads, bit for bit: the
tabulated factors toDose / rho and the corrected quotient by the history count are the
doubles that divisions give.  Odd and even voxel counts, one voxel, voxels without events
or density, spacings that leave the table's range, and output arrays off a 16-byte boundary
(one voxel a thread) or on it (two)."""
import numpy as np
import pytest

from opendxmc_gb300 import phantoms as P

pytestmark = pytest.mark.gpu

KEV_TO_MGY_G = 1.602176634e-10


def reference(world, spacing, n_hist):
    e, e2, c = world.tally()
    rho = world.packed_density()[0].astype(np.float64)
    vol = spacing[0] * spacing[1] * spacing[2]
    s = np.divide(KEV_TO_MGY_G / vol, rho, out=np.zeros_like(rho), where=rho > 0)
    v = e2 - e * e / n_hist if n_hist else np.zeros_like(e)
    return e * s, np.where(v > 0, v, 0.0) * s * s, c


@pytest.mark.parametrize("dims,spacing,hist", [
    ((1, 1, 1), (9.0, 9.0, 9.0), 5000), ((7, 5, 3), (1.0, 1.5, 2.0), 20_000), ((33, 17, 9), (0.3, 0.4, 0.5), 100_000),
    ((32, 16, 10), (0.3, 0.4, 0.5), 3), ((6, 5, 4), (1e-80, 1e-80, 1e-80), 100)])
@pytest.mark.parametrize("shift", [0, 1])
def test_readout_is_the_plain_formula(gpu, dims, spacing, hist, shift):
    rng = np.random.default_rng(sum(dims))
    n = int(np.prod(dims))
    # densities over several octaves, zero among them
    rho = (rng.uniform(0.0, 1.0, n) * 2.0 ** rng.integers(-6, 4, n)).astype(np.float32)
    rho[rng.random(n) < 0.1] = 0.0
    w = gpu.GpuWorld(dims, spacing, [P.WATER])
    w.set_data(rho, np.zeros(n, np.uint8))
    w.build()
    beam = P.dx_beam_params(field_cm=2.0, particles=hist, exposures=1)
    done = w.run(beam, gpu.run_options(seed=4))["n_histories"]
    arrays = [np.full(n + 2, 7, t) for t in (np.float64, np.float64, np.uint64)]
    # this library's host staging is read back into the arrays whatever their alignment; the
    # kernel's own scalar path is reached through pinned arrays off the boundary
    import torch

    pinned = [torch.from_numpy(a.view(np.int64) if a.dtype == np.uint64 else a).pin_memory().numpy() for a in arrays]
    start = [(-x.ctypes.data // 8) % 2 + shift for x in pinned]
    out = [x[k:k + n] for x, k in zip(pinned, start)]
    assert all((x.ctypes.data % 16 == 8) == bool(shift) for x in out)
    d, v, c = w.dose(out=(out[0], out[1], out[2].view(np.uint64)))
    rd, rv, rc = reference(w, spacing, done)
    np.testing.assert_array_equal(d, rd)
    np.testing.assert_array_equal(v, rv)
    np.testing.assert_array_equal(c, rc)
    for x, k in zip(pinned, start):  # nothing written beside the arrays
        assert (np.delete(x, np.arange(k, k + n)) == 7).all()
    if n > 1:
        assert (rc == 0).any() or hist > 1000
