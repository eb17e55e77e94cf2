"""The Woodcock kernel's photon pools and shared attenuation tables: which lane and phase does
a history's work, and where its tables lie, changes nothing of the history."""
import numpy as np
import pytest

from opendxmc_gb300 import phantoms as P

pytestmark = pytest.mark.gpu

COUNTS = ("n_histories", "n_visits", "n_photo", "n_compton", "n_rayleigh", "n_cutoff", "n_interacted", "n_missed")
MATERIALS = [P.AIR, P.WATER, P.BONE]


def world(gpu, mat, dens, materials, correction=1):
    nz, ny, nx = mat.shape
    w = gpu.GpuWorld((nx, ny, nz), (0.7, 0.9, 1.1), materials, correction)
    w.set_data(dens, mat)
    w.build()
    return w


def volume(copies):
    """Three materials with transparent and empty voxels; with `copies`, material m also goes
    by the indices m + 3, m + 6, ..."""
    rng = np.random.default_rng(5)
    base = rng.integers(0, 3, (11, 13, 17))
    dens = np.array([0.0012, 1.0, 1.92])[base] * rng.uniform(0.9, 1.1, base.shape)
    dens.ravel()[::11] = 0.0
    mat = (base + 3 * rng.integers(0, copies, base.shape)).astype(np.uint8)
    mat[4:6, 5:8, 2:9] = 255
    return mat, dens


def outcome(w, gpu, histories, correction, **options):
    beam = P.dx_beam_params(particles=histories, exposures=1, field_cm=16.0)
    w.clear()
    s = w.run(beam, gpu.run_options(seed=4, stream=2, **options))
    assert s["n_errors"] == 0 and s["n_histories"] == histories
    return s, w.tally()


def same(a, b):
    for k in COUNTS:
        assert a[0][k] == b[0][k], k
    np.testing.assert_array_equal(a[1][2], b[1][2])
    for x, y in zip(a[1][:2], b[1][:2]):  # FP64 atomics in another order
        np.testing.assert_allclose(x, y, rtol=1e-12, atol=0)


@pytest.mark.parametrize("correction", [1, 2])
@pytest.mark.parametrize("histories", [1, 31, 65, 20_000])
def test_phases_and_tables_leave_histories_alone(gpu, histories, correction):
    """One photon, less and little more than a warp's pool, and many; the batches at their
    ends; six materials with the tables in shared memory and nine without."""
    mat, dens = volume(1)
    w = world(gpu, mat, dens, MATERIALS, correction)
    ref = outcome(w, gpu, histories, correction)
    for two in (-1, 1):
        plain = outcome(w, gpu, histories, correction, two_region=two)
        for o in ({"interact_batch": 1, "refill_batch": 1, "woodcock_steps": 1},
                  {"interact_batch": 32, "refill_batch": 32, "woodcock_steps": 64}):
            same(outcome(w, gpu, histories, correction, two_region=two, **o), plain)
    for copies in (2, 3):  # 6 and 9 materials
        m, d = volume(copies)
        np.testing.assert_array_equal(d, dens)
        same(outcome(world(gpu, m, d, MATERIALS * copies, correction), gpu, histories, correction), ref)
