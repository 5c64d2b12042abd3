"""The FP64 sums' tiles against the oracle, bit for bit: ring counts and target
counts about the batch and tile sizes, and wake sheets whose rows and stations
are shorter than, equal to and longer than a batch, with summation blocks that
end inside columns."""
import numpy as np
import pytest

from oracle import oracle as O
from volcanor_gb300 import cases as C
from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (3, 1), (128, 2), (129, 31), (257, 33), (700, 129), (2049, 7), (40, 20001)])
def test_rings_bitwise(n, m):
    rng = np.random.default_rng(n + m)
    corners = rng.uniform(size=(n, 1, 3)) + 0.05 * rng.uniform(size=(n, 4, 3))
    rvc, gam, P = rng.uniform(0, 0.01, (n, 4)), rng.normal(size=n), rng.uniform(size=(m, 3))
    gam[::7] = 0.0
    P[0] = corners[0, 1]  # a target on a corner
    chunk = lib.rings_sum_chunk(n, m)
    np.testing.assert_array_equal(lib.biot_savart_rings(corners, rvc, gam, P),
                                  O.vind_rings(corners, rvc, gam, P, chunk=chunk if chunk < n else 0))


# (blades, stations, near-wake rows, truncation, steps, summation block)
@pytest.mark.parametrize("nb,ns,rows,trunc,steps,chunk", [
    (1, 1, 3, 5, 8, 2),       # one column: no neighbour across, rows far below a batch
    (2, 3, 2, 5, 7, 256),     # two rows, the fewest a case takes
    (2, 24, 9, 13, 18, 64),   # a batch spans columns
    (1, 2, 300, 0, 290, 256), # columns longer than a batch of one target
    (3, 11, 40, 46, 52, 37),  # blocks that end inside columns
])
def test_sheets_bitwise(nb, ns, rows, trunc, steps, chunk):
    cfg = C.config_text(nt=steps, dt=0.0, density=1.2, kinematicVisc=1.5e-5, fdScheme=3, wakeDissipation=1)
    geo = C.geom_text(nb=nb, nc=1, ns=ns, nNwake=rows, span=1.0, rootcut=0.2, chord=0.08, Omega=100.0,
                      shaftAxis=(0.0, 0.0, 1.0), theta0=8.0, velBody=(-8.0, 0.0, 0.0), spanSpacing=1, chordSpacing=1,
                      spanwiseCore=0.05, streamwiseCoreVec=0.05, apparentViscCoeff=5.0, wakeTruncateNt=trunc,
                      symmetricTau=0, pivotLE=0.25)
    g = lib.Case(cfg, geo, precision=lib.PREC_FP64, sum_chunk=chunk)
    g.start()
    g.step(steps)
    r = O.Sim(cfg, geo)
    r.set_sum_chunk(chunk)
    r.start()
    r.step(steps)
    np.testing.assert_array_equal(g.ct_hist(), r.ct_hist())
    for b in range(1, nb + 1):
        np.testing.assert_array_equal(g.get("waN", b).reshape(-1, 4, 3), r.get("waN", b).reshape(-1, 4, 2, 3)[:, :, 0])
        np.testing.assert_array_equal(g.get("waF", b), r.get("waF", b))
