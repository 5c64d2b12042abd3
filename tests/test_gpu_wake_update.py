"""The wake update (shedding, ageing, dissipation, predictor, corrector, strain,
rollup, row moves) against the oracle, bit for bit, from the first rows to a full
wake, at its edges: two rows and one station, a far wake of one and two
filaments, more blades than one block rolls up, and no far wake."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_solver import assert_same_state
from volcanor_gb300 import cases as C
from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fd,nb,ns,rows,trunc,strain", [(3, 1, 1, 2, 3, 1), (1, 2, 3, 3, 5, 0), (3, 5, 9, 4, 9, 1),
                                                        (5, 2, 33, 5, 7, 1), (4, 1, 4, 6, 0, 0)])
def test_wake_update_bitwise(fd, nb, ns, rows, trunc, strain):
    steps = max(trunc, rows) + 4
    cfg = C.config_text(nt=steps, dt=0.0, density=1.2, kinematicVisc=1.5e-5, fdScheme=fd, wakeDissipation=1,
                        wakeStrain=strain)
    geo = C.geom_text(nb=nb, nc=1, ns=ns, nNwake=rows, span=1.0, rootcut=0.2, chord=0.08, Omega=100.0,
                      shaftAxis=(0.0, 0.0, 1.0), theta0=8.0, velBody=(-8.0, 0.0, 0.0), spanSpacing=1, chordSpacing=1,
                      spanwiseCore=0.05, streamwiseCoreVec=0.05, apparentViscCoeff=5.0, wakeTruncateNt=trunc,
                      symmetricTau=0, pivotLE=0.25, rollupStartRadius=0.5, rollupEndRadius=1.0)
    g = lib.Case(cfg, geo, precision=lib.PREC_FP64, sum_chunk=64)
    r = O.Sim(cfg, geo)
    r.set_sum_chunk(64)
    g.start()
    r.start()
    for _ in range(steps):
        g.step(1)
        r.step(1)
        assert_same_state(g, r, nb)
    np.testing.assert_array_equal(g.ct_hist(), r.ct_hist())
