"""The line plans whose lines do not fill a warp evenly (400, 432, 720 points:
20, 36 and 24 lanes) and the other plans beside the power-of-two ones, against
the block engine and cuFFT on one exact deposit."""
import pytest

from helpers import particle_set, rel_rms
from test_gravity_long_gpu import device_phi
from tigerpm_b200.api import GRAVITY_LONG_PM, GRAVITY_LONG_PME

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("typ", [GRAVITY_LONG_PME, GRAVITY_LONG_PM])
@pytest.mark.parametrize("grid", [48, 80, 400, 432, 480, 720])
def test_line_plan(grid, typ):
    ps = particle_set("uniform", 24, 6)
    phi, _ = device_phi(ps, grid, "cloud4", 2.0, typ, exact=True)
    for other in ("block", "cufft"):
        ref, _ = device_phi(ps, grid, "cloud4", 2.0, typ, exact=True, fft=other)
        # FP32 transforms of different radix orders (the tolerance of the other line plans)
        assert rel_rms(phi, ref) < 2e-6, (other, rel_rms(phi, ref))
