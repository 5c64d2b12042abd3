"""Near-field pairs of ring sums at the sizes where their search changes:
below, at and above a tile of targets, few rings at many targets, and on both
sides of the limit between testing every pair and the target grid (2^24 pairs).

Square rings of 0.03 with core radius 0.05, 10 apart, targets about their
centres: all four filaments of the target's own ring are near (4 core radii)
and add up without cancellation, every other ring's velocity is below 1e-7 of
theirs.  Corrected, what is left is the rounding of the four terms in the FP32
sums (4 x 6e-8); a filament missed keeps its FP32 position error, up to 8e-6
(coordinates to 160) in 0.015, a quarter of the sum: above 1e-5 in the median
of the targets of the outer rings, so each target is held to 2e-6."""
import numpy as np
import pytest

from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (1, 63), (3, 64), (129, 65), (4096, 129), (40, 70001), (4096, 4096), (4097, 4096)])
def test_near_pairs(n, m):
    rng = np.random.default_rng(n + m)
    c = 10.0 * np.stack(np.unravel_index(np.arange(n), (17, 17, 17)), axis=1) + rng.uniform(0, 1, size=(n, 3))
    sq = 0.015 * np.array([[-1, -1, 0], [1, -1, 0], [1, 1, 0], [-1, 1, 0]])
    corners = c[:, None] + sq
    P = c[(np.arange(m) * 7919) % n] + rng.uniform(-0.003, 0.003, size=(m, 3))
    rvc, gam = np.full((n, 4), 0.05), rng.uniform(1, 2, n)
    V64 = lib.biot_savart_rings(corners, rvc, gam, P, lib.PREC_FP64)
    err = np.linalg.norm(lib.biot_savart_rings(corners, rvc, gam, P, lib.PREC_FP32_NEAR64) - V64, axis=1)
    assert (err / np.linalg.norm(V64, axis=1)).max() < 2e-6
