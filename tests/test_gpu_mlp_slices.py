"""The MLP gradient at batch sizes about the slice and tile sizes and at ragged
layer widths, against the FP64 oracle (1e-4 of the gradient's norm, the bound of
the gradient test at one size)."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO
from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 1), (12, 128, 128, 3), (5, 65, 129, 2), (3, 200, 4)])
@pytest.mark.parametrize("n", [1, 16, 127, 128, 129, 300, 8200])
def test_gradient_against_oracle(sizes, n):
    rng = np.random.default_rng(n)
    net = lib.Mlp(list(sizes), seed=n)
    X = rng.uniform(-1, 1, (n, sizes[0])).astype(np.float32)
    T = rng.normal(size=(n, sizes[-1])).astype(np.float32)
    g, loss = net.gradient(X, T)
    want, want_loss = MO.gradient(net.get_params().astype(np.float64), list(sizes), X, T)
    assert np.linalg.norm(g - want) <= 1e-4 * np.linalg.norm(want)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    again, _ = net.gradient(X, T)
    np.testing.assert_array_equal(g, again)
