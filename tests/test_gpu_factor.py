"""The AIC's FP64 inverse against the oracle, bit for bit, at panel counts about
the factorisation's panel and tile sizes (1, 15, 16, 17, 31 .. 150 rows), and the
refined FP32 solve's residual there."""
import numpy as np
import pytest

from oracle import oracle as O
from volcanor_gb300 import cases as C
from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


def case(nb, nc, ns):
    cfg = C.config_text(nt=2, dt=0.002, density=1.2, kinematicVisc=1.5e-5, fdScheme=3)
    geo = C.geom_text(nb=nb, nc=nc, ns=ns, nNwake=2, span=1.0, rootcut=0.2, chord=0.08, Omega=100.0,
                      shaftAxis=(0.0, 0.0, 1.0), theta0=8.0, velBody=(-8.0, 0.0, 1.0), spanSpacing=1, chordSpacing=1,
                      spanwiseCore=0.05, streamwiseCoreVec=0.05, apparentViscCoeff=5.0, symmetricTau=0, pivotLE=0.25)
    return cfg, geo


@pytest.mark.parametrize("nb,nc,ns", [(1, 1, 1), (1, 3, 5), (2, 1, 8), (1, 1, 17), (1, 1, 31), (2, 4, 4), (3, 1, 11),
                                      (2, 1, 64), (3, 2, 25)])
def test_inverse_bitwise_and_refined_solve(nb, nc, ns):
    cfg, geo = case(nb, nc, ns)
    g, r = lib.Case(cfg, geo, precision=lib.PREC_FP64), O.Sim(cfg, geo)
    g.start()
    r.start()
    np.testing.assert_array_equal(g.get("AIC"), r.get("AIC"))
    np.testing.assert_array_equal(g.get("AIC_inv"), r.get("AIC_inv"))
    np.testing.assert_array_equal(g.get("gamVec"), r.get("gamVec"))
    f = lib.Case(cfg, geo, precision=lib.PREC_FP32)
    f.start()
    assert f.get("lu_residual")[0] < 1e-12
    np.testing.assert_allclose(f.get("gamVec"), r.get("gamVec"), rtol=0, atol=1e-11 * np.abs(r.get("gamVec")).max())
