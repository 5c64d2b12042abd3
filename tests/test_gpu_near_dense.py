"""Near-field pairs by the thousand: 128 rings about one point, all of whose
filaments are near all the targets there, are one block's work (4096 pairs for 8
targets), more than its buffer of 768 takes; with circulations of 1e5 the
corrections, about 1e-4 of a filament's velocity of 4 times its circulation, are
beyond the 64 up to which they are added as integers.

The rings lie about parallel and turn the same way, so their velocities add up.
What the corrections leave is the rounding of the FP32 sums, 512 terms of one sign
for a tile: at most 512 x 2^-24 = 3.1e-5 of the sum, which is the bound.  At
100 from the origin a target's FP32 position is off by up to 3.8e-6, the same for
all its terms; 0.01 above rings of half width 0.015 that changes the velocity by
up to 3.8e-6 / 0.02 = 1.9e-4, so uncorrected pairs show."""
import numpy as np
import pytest

from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gam", [1.0, 1e5])
@pytest.mark.parametrize("m", [8, 64, 300])
def test_every_pair_near(m, gam):
    rng = np.random.default_rng(m)
    at = np.array([100.0, 90.0, 80.0])
    sq = 0.015 * np.array([[-1, -1, 0], [1, -1, 0], [1, 1, 0], [-1, 1, 0]])
    corners = at + sq + rng.uniform(-5e-4, 5e-4, size=(128, 4, 3))
    P = at + np.array([0.0, 0.0, 0.01]) + rng.uniform(-0.002, 0.002, size=(m, 3))
    rvc, g = np.full((128, 4), 0.02), gam * rng.uniform(1, 2, 128)
    V64 = lib.biot_savart_rings(corners, rvc, g, P, lib.PREC_FP64)
    size = np.linalg.norm(V64, axis=1)
    near = np.linalg.norm(lib.biot_savart_rings(corners, rvc, g, P, lib.PREC_FP32_NEAR64) - V64, axis=1) / size
    assert near.max() < 3.1e-5
    if m == 300:  # the bound tells corrected from uncorrected sums
        far = np.linalg.norm(lib.biot_savart_rings(corners, rvc, g, P, lib.PREC_FP32) - V64, axis=1) / size
        assert far.max() > 2 * 3.1e-5
