"""Bias gradients of a training step: a CTA's sums are added in FP64, so the order
of the CTAs does not show (FP32 atomics before, several digits apart)."""
import numpy as np
import pytest

import bbpp
from bbpp import learned

pytestmark = pytest.mark.gpu
LAYERS = [(16, 16), (16, 32), (32, 64), (96, 32), (48, 16)]


@pytest.mark.parametrize("n,nb", [(8, 1), (32, 1), (48, 3), (64, 4)])
def test_bias_gradients_do_not_depend_on_the_order(bbpp_lib, n, nb):
    rng = np.random.default_rng(n)
    d = [bbpp.DeviceArray.from_host(rng.standard_normal((nb, n, n, n)).astype(np.float32)) for _ in range(3)]
    net = learned.Net(seed=3)
    runs = [net.loss_grad((n, n, n), 1.0 / n ** 2, *d)[1] for _ in range(6)]
    off = 0
    for cin, cout in LAYERS:
        off += 27 * cin * cout
        b = [g[off:off + cout] for g in runs]
        assert np.any(b[0] != 0)
        for other in b[1:]:
            # FP64 sums round to neighbouring floats at most
            assert np.all(np.abs(b[0] - other) <= np.spacing(np.abs(b[0])))
        off += cout
