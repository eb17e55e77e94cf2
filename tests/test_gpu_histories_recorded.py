"""The transport's histories against those that the one-photon-a-lane Woodcock kernel, the
predecessor of the photon pools, gave for the same seeds: event counts, and a checksum of the
events in every voxel.  Correction levels 1 and 2 (with iodine), one and two regions, with and
without cell bounds, and the other tracking modes.  The counts hold for this library's host
tables, whose FP64 logarithms and powers come from the C library."""
import numpy as np
import pytest

from opendxmc_gb300 import native as N
from opendxmc_gb300 import phantoms as P

pytestmark = pytest.mark.gpu

MATERIALS = [P.AIR, P.WATER, P.BONE, {1: 10.0, 8: 85.0, 53: 5.0}]
COUNTS = ("n_missed", "n_visits", "n_photo", "n_compton", "n_rayleigh", "n_cutoff", "n_fluorescence", "n_interacted")

# (tracking, correction, gather_skip, two_region)
CASES = [(N.TRACK_WOODCOCK, c, s, t) for c in (1, 2) for s in (-1, 1) for t in (-1, 1)] \
    + [(m, c, 0, 0) for m in (N.TRACK_SIDDON, N.TRACK_MACRO) for c in (1, 2)]


def outcome(gpu, tracking, correction, skip, two):
    rng = np.random.default_rng(11)
    mat = np.zeros((21, 33, 40), np.uint8)
    inner = mat[3:17, 5:26, 8:33]
    inner[:] = rng.integers(0, 4, inner.shape)
    dens = np.array([0.0012, 1.0, 1.92, 1.1])[mat] * rng.uniform(0.9, 1.1, mat.shape)
    dens.ravel()[::13] = 0.0
    mat[9:11, 12:15, 20:24] = 255
    w = gpu.GpuWorld((40, 33, 21), (0.5, 0.6, 0.9), MATERIALS, correction)
    w.set_data(dens, mat)
    w.build()
    beam = P.dx_beam_params(kvp=120.0, particles=400_000, exposures=1, field_cm=18.0)
    s = w.run(beam, gpu.run_options(seed=9, stream=1, tracking=tracking, gather_skip=skip, two_region=two))
    assert s["n_errors"] == 0 and s["n_histories"] == 400_000
    c = w.tally()[2].astype(np.int64)
    return [int(s[k]) for k in COUNTS] + [int((c * (np.arange(c.size) % 65_521 + 1)).sum())]


RECORDED = {
    (N.TRACK_WOODCOCK, 1, -1, -1): [0, 7423551, 157225, 141815, 21730, 0, 0, 200957, 4003927688],
    (N.TRACK_WOODCOCK, 1, -1, 1): [0, 868494, 157642, 140849, 21753, 0, 0, 201199, 3994421511],
    (N.TRACK_WOODCOCK, 1, 1, -1): [0, 7423551, 157225, 141815, 21730, 0, 0, 200957, 4003927688],
    (N.TRACK_WOODCOCK, 1, 1, 1): [0, 868494, 157642, 140849, 21753, 0, 0, 201199, 3994421511],
    (N.TRACK_WOODCOCK, 2, -1, -1): [0, 7760860, 201534, 151823, 26512, 0, 52763, 200957, 4728455752],
    (N.TRACK_WOODCOCK, 2, -1, 1): [0, 1064237, 201765, 151106, 26552, 0, 52495, 201199, 4719908526],
    (N.TRACK_WOODCOCK, 2, 1, -1): [0, 7760860, 201534, 151823, 26512, 0, 52763, 200957, 4728455752],
    (N.TRACK_WOODCOCK, 2, 1, 1): [0, 1064237, 201765, 151106, 26552, 0, 52495, 201199, 4719908526],
    (N.TRACK_SIDDON, 1, 0, 0): [0, 11100324, 157710, 141029, 21671, 0, 0, 201076, 4000143348],
    (N.TRACK_SIDDON, 2, 0, 0): [0, 11426761, 201959, 150917, 26589, 0, 52659, 201076, 4722089834],
    (N.TRACK_MACRO, 1, 0, 0): [0, 7052938, 157761, 141782, 21751, 0, 0, 201053, 4006990265],
    (N.TRACK_MACRO, 2, 0, 0): [0, 7381382, 201207, 152005, 26596, 0, 52265, 201053, 4727102442],
}


@pytest.mark.parametrize("case", CASES)
def test_histories_are_those_recorded(gpu, case):
    assert outcome(gpu, *case) == RECORDED[case]
