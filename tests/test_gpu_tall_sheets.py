"""FP64 sums over wake sheets about the heights where the tile of a block
changes: above 1488 rows an SM holds one block instead of two, above 3909 a
column's edges no longer fit shared memory and the rings are summed one by one.
An FP32 run makes the wake, the FP64 form and the oracle take its state over
and make one step: bit for bit the same."""
import numpy as np
import pytest

from oracle import handoff
from oracle import oracle as O
from volcanor_gb300 import cases as C
from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1488, 1489, 3909, 3910])
def test_step_bitwise(rows, tmp_path):
    cfg = C.config_text(nt=rows, dt=0.025, density=1.0, kinematicVisc=1.5e-5, fdScheme=3, wakeDissipation=1)
    geo = C.geom_text(nb=1, nc=1, ns=2, nNwake=rows, span=4.0, rootcut=0.0, chord=1.0, Omega=0.0, theta0=5.0,
                      velBody=(-10.0, 0.0, 0.0), spanSpacing=1, chordSpacing=1, spanwiseCore=0.03,
                      streamwiseCoreVec=0.03, apparentViscCoeff=5.0, symmetricTau=1)
    path = str(tmp_path / "wake.ckpt")
    f = lib.Case(cfg, geo, precision=lib.PREC_FP32)
    f.start()
    f.step(rows - 1)
    f.checkpoint_save(path)
    f.close()
    g = lib.Case(cfg, geo, precision=lib.PREC_FP64, sum_chunk=256)
    g.start()
    g.checkpoint_load(path)
    O.set_threads(16)
    r = O.Sim(cfg, geo)
    r.set_sum_chunk(256)
    r.start()
    handoff.load_case_state(r, g)
    g.step(1)
    r.step(1)
    np.testing.assert_array_equal(g.ct_hist()[-1], r.ct_hist()[-1])
    np.testing.assert_array_equal(g.get("waN").reshape(-1, 4, 3), r.get("waN").reshape(-1, 4, 2, 3)[:, :, 0])
    np.testing.assert_array_equal(g.get("velN"), r.get("velN"))
