"""The collocation points' total velocities (ring and bound-vortex sums of the
wing) against the oracle, bit for bit through the loads: one blade in several
batches of 256 rings, several blades in one, more blades than a group of 32
takes, and one to several chordwise panels, whose rings share corners and edges."""
import numpy as np
import pytest

from oracle import oracle as O
from volcanor_gb300 import cases as C
from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,nc,ns,chunk", [(1, 1, 1, 256), (3, 1, 5, 2), (5, 4, 20, 256), (1, 16, 20, 100), (2, 9, 30, 256),
                                            (34, 1, 2, 256)])
def test_loads_bitwise(nb, nc, ns, chunk):
    steps = 3
    cfg = C.config_text(nt=steps, dt=0.0, density=1.2, kinematicVisc=1.5e-5, fdScheme=3, wakeDissipation=1)
    geo = C.geom_text(nb=nb, nc=nc, ns=ns, nNwake=4, span=1.0, rootcut=0.2, chord=0.08, Omega=100.0,
                      shaftAxis=(0.0, 0.0, 1.0), theta0=8.0, velBody=(-8.0, 0.0, 0.0), spanSpacing=1, chordSpacing=1,
                      spanwiseCore=0.05, streamwiseCoreVec=0.05, apparentViscCoeff=5.0, wakeTruncateNt=6,
                      symmetricTau=0, pivotLE=0.25)
    g = lib.Case(cfg, geo, precision=lib.PREC_FP64, sum_chunk=chunk)
    g.start()
    g.step(steps)
    r = O.Sim(cfg, geo)
    r.set_sum_chunk(chunk)
    r.start()
    r.step(steps)
    np.testing.assert_array_equal(g.ct_hist(), r.ct_hist())
