"""The transport's own arithmetic forms against CUDA's functions, bit for bit over every float of
their ranges, and its bound-electron samplers against their plain loops on the same uniforms
(tests/cpp/arithmetic.cu, built here)."""
import subprocess
from pathlib import Path

import pytest

from opendxmc_gb300 import build as B

pytestmark = pytest.mark.gpu

SOURCE = Path(__file__).parent / "cpp" / "arithmetic.cu"


@pytest.fixture(scope="module")
def checks(gpu, tmp_path_factory):
    exe = tmp_path_factory.mktemp("arithmetic") / "arithmetic"
    r = subprocess.run([B.nvcc(), *B.ARCH, *B.COMMON, str(SOURCE), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return {name: (int(bad), int(total)) for name, bad, _, total in (line.split() for line in r.stdout.splitlines())}


@pytest.mark.parametrize("name,total", [
    ("reciprocal", 219 << 23), ("squareRoot", 209 << 23), ("squareRootOfZero", 1), ("unitRsqrt", 4 << 23),
    ("negLog", 1 << 23), ("dopplerEnergyFused", 1 << 23), ("dopplerEnergyPlain", 1 << 23),
    ("samplePhotoFluorescenceFused", 1 << 23), ("samplePhotoFluorescencePlain", 1 << 23)])
def test_same_bits(checks, name, total):
    assert checks[name] == (0, total)


def test_bound_electron_draws_are_taken_and_refused(checks):
    taken, total = checks["takenFused"]
    assert 0.2 * total < taken < 0.98 * total
