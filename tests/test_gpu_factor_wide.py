"""AIC factors and solves of wide matrices: LU panels of fewer than 16 columns
(above 1808 rows in FP64, 3616 in FP32) and the refined solve with more than the
default shared memory (above 2680 rows).

FP64: the inverse bit for bit against the same operations in numpy, at every
29th column.  FP32: the refined circulations against those of the FP64 inverse,
within the normwise error of a solve, n 2^-53 times the condition number, twice
over for either side."""
import numpy as np
import pytest

from volcanor_gb300 import cases as C
from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


def case(nc, ns, precision):
    cfg = C.config_text(nt=2, dt=0.002, density=1.2, kinematicVisc=1.5e-5, fdScheme=3)
    geo = C.geom_text(nb=1, nc=nc, ns=ns, nNwake=2, span=8.0, rootcut=0.1, chord=0.5, Omega=100.0,
                      shaftAxis=(0.0, 0.0, 1.0), theta0=8.0, velBody=(-8.0, 0.0, 1.0), spanSpacing=1, chordSpacing=1,
                      spanwiseCore=0.05, streamwiseCoreVec=0.05, apparentViscCoeff=5.0, symmetricTau=0, pivotLE=0.25)
    c = lib.Case(cfg, geo, precision=precision)
    c.start()
    return c


def inverse_columns(A, cols):
    """LU with partial pivoting, then the identity's columns forward and backward, every
    element updated by k = 0, 1, ... in turn and each operation rounded."""
    n = A.shape[0]
    A, X = A.copy(), np.eye(n)[:, cols]
    for k in range(n):
        p = k + int(np.argmax(np.abs(A[k:, k])))
        A[[k, p]], X[[k, p]] = A[[p, k]], X[[p, k]]
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= A[k + 1:, k, None] * A[k, k + 1:]
    for k in range(n):
        X[k + 1:] -= A[k + 1:, k, None] * X[k]
    for i in range(n - 1, -1, -1):
        X[i] = np.subtract.reduce(np.concatenate([X[i:i + 1], A[i, i + 1:, None] * X[i + 1:]]), axis=0) / A[i, i]
    return X


def test_inverse_bitwise():
    c = case(4, 453, lib.PREC_FP64)
    n = 4 * 453
    cols = np.arange(0, n, 29)
    np.testing.assert_array_equal(c.get("AIC_inv").reshape(n, n).T[:, cols],
                                  inverse_columns(c.get("AIC").reshape(n, n).T, cols))


@pytest.mark.parametrize("nc,ns", [(4, 453), (10, 280), (10, 370)])
def test_refined_solve(nc, ns):
    c = case(nc, ns, lib.PREC_FP32)
    n = nc * ns
    kappa = np.linalg.norm(c.get("AIC").reshape(n, n), 1) * np.linalg.norm(c.get("AIC_inv").reshape(n, n), 1)
    x = case(nc, ns, lib.PREC_FP64).get("gamVec")
    assert c.get("lu_residual")[0] < 1e-9
    assert np.abs(c.get("gamVec") - x).max() <= 4 * n * 2.0 ** -53 * kappa * np.abs(x).max()
