"""Host-buffer ring and filament sums against the device-buffer calls, bit for
bit: sizes on both sides of the packed-copy limit (2 MiB of arrays), larger
and smaller calls in turn, and no sources at all."""
import numpy as np
import pytest

from volcanor_gb300 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [lib.PREC_FP64, lib.PREC_FP32_NEAR64])
def test_host_equals_device_call(precision):
    import torch

    rng = np.random.default_rng(precision)
    for n, m in [(1, 1), (15400, 40), (15420, 40), (52, 52), (0, 5), (15440, 40), (33, 43000), (33, 1)]:
        corners = rng.uniform(size=(n, 1, 3)) + 0.05 * rng.uniform(size=(n, 4, 3))
        rvc, gam, P = rng.uniform(0, 0.01, (n, 4)), rng.normal(size=n), rng.uniform(size=(m, 3))
        t = [torch.from_numpy(a).cuda() for a in (corners, rvc, gam, P)]
        V = torch.full((m, 3), 7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        lib.biot_savart_rings_device(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), n, t[3].data_ptr(), m,
                                     V.data_ptr(), precision)
        np.testing.assert_array_equal(lib.biot_savart_rings(corners, rvc, gam, P, precision), V.cpu().numpy())
        if n == 0:
            np.testing.assert_array_equal(V.cpu().numpy(), 0.0)
