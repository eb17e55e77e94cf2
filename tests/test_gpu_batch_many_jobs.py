"""Batches of many small jobs, which share launches: each job's histories are those of its run
alone, whatever kernel instance it needs and however many jobs there are; and the batch takes
about as long as its work, not as long as its jobs' longest histories one after another."""
import numpy as np
import pytest

from opendxmc_gb300 import native as N
from opendxmc_gb300 import phantoms as P

pytestmark = pytest.mark.gpu

MATERIALS = [P.AIR, P.WATER, P.BONE]
COUNTS = ("n_histories", "n_missed", "n_visits", "n_photo", "n_compton", "n_rayleigh", "n_fluorescence",
          "n_interacted")


def make_worlds(gpu):
    """Grids with one and two regions, attenuation tables in shared memory (3 and 6 materials)
    and not (9), correction levels 1 and 2."""
    worlds = []
    for k, (dims, copies, correction) in enumerate([((23, 17, 11), 1, 1), ((40, 32, 24), 2, 1), ((31, 33, 19), 3, 1),
                                                    ((32, 16, 16), 1, 2), ((28, 30, 21), 3, 2)]):
        rng = np.random.default_rng(k)
        nx, ny, nz = dims
        mat = np.zeros((nz, ny, nx), np.uint8)
        inner = mat[2:nz - 3, 3:ny - 4, 4:nx - 6]
        inner[:] = rng.integers(0, 3 * copies, inner.shape)
        dens = np.array([0.0012, 1.0, 1.92])[mat % 3] * rng.uniform(0.9, 1.1, mat.shape)
        w = gpu.GpuWorld(dims, (0.7, 0.8, 0.9), MATERIALS * copies, correction)
        w.set_data(dens, mat)
        w.build()
        worlds.append(w)
    return worlds


@pytest.mark.parametrize("tracking,jobs,histories,skip", [
    (N.TRACK_WOODCOCK, 2, 60, 0), (N.TRACK_WOODCOCK, 64, 500, 0), (N.TRACK_WOODCOCK, 333, 700, 0),
    (N.TRACK_WOODCOCK, 333, 700, 1), (N.TRACK_SIDDON, 130, 500, 0), (N.TRACK_MACRO, 130, 500, 0),
    (N.TRACK_SIDDON, 130, 15_000, 0), (N.TRACK_MACRO, 130, 15_000, 0)])  # the last two: one queue
def test_histories_are_those_of_the_jobs_alone(gpu, tracking, jobs, histories, skip):
    worlds, twins = make_worlds(gpu), make_worlds(gpu)
    rng = np.random.default_rng(jobs + histories)
    plan = []
    for j in range(jobs):
        w = int(rng.integers(len(worlds)))
        beam = P.dx_beam_params(kvp=60.0 + j % 70, field_cm=16.0, particles=int(rng.integers(1, histories)), exposures=1)
        plan.append((w, beam, dict(seed=j, stream=j % 3, tracking=tracking, gather_skip=skip,
                                   two_region=int(rng.integers(-1, 2)) if tracking == N.TRACK_WOODCOCK else 0,
                                   block_size=int(rng.choice([0, 0, 64])))))
    batch = gpu.Batch([(worlds[w], beam, gpu.run_options(**o)) for w, beam, o in plan])
    got = batch.run()
    total = dict.fromkeys(COUNTS, 0)
    for w, beam, o in plan:
        s = twins[w].run(beam, gpu.run_options(**o))
        for k in COUNTS:
            total[k] += s[k]
    assert got["n_errors"] == 0
    assert {k: got[k] for k in COUNTS} == total
    for repeat in (1, 2):
        for a, b in zip(worlds, twins):
            np.testing.assert_array_equal(a.tally()[2], repeat * b.tally()[2])
            np.testing.assert_allclose(a.tally()[0], repeat * b.tally()[0], rtol=1e-12)
        if repeat == 1:
            batch.run()
    batch.close()


@pytest.mark.parametrize("tracking", [N.TRACK_WOODCOCK, N.TRACK_SIDDON, N.TRACK_MACRO])
def test_many_jobs_run_together(gpu, tracking):
    """512 jobs of 1000 histories fit the device at once, as 32 do: less than five times as long
    (measured 1.2 to 2.7 times; 9 to 15 with a launch a job)."""
    ph = P.ellipsoid_phantom((64, 64, 64), (0.3, 0.3, 0.3), seed=3)
    w = gpu.GpuWorld(ph.dims, ph.spacing, ph.materials)
    w.set_data(ph.density, ph.material)
    w.build()
    beam = P.dx_beam_params(particles=1000, exposures=1)
    ms = []
    for jobs in (32, 512):
        batch = gpu.Batch([(w, beam, gpu.run_options(seed=j, tracking=tracking)) for j in range(jobs)])
        ms.append(min(batch.run()["kernel_ms"] for _ in range(6)))
        batch.close()
    assert ms[1] < 5.0 * ms[0], ms
