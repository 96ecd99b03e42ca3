"""The weight gradient with several tiles a CTA (its two stages alternate), on
partial tiles, against an FP64 convolution gradient."""
import numpy as np
import pytest

import bbpp
from bbpp import learned
import net_oracle as NO

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,dims,nb", [(16, 16, (64, 64, 33), 3), (48, 16, (63, 50, 30), 2),
                                              (96, 32, (48, 41, 32), 2), (16, 32, (64, 64, 33), 2),
                                              (32, 64, (50, 48, 31), 2)])
def test_wgrad_many_tiles(bbpp_lib, cin, cout, dims, nb):
    L = learned._sig()
    nx, ny, nz = dims
    rng = np.random.default_rng(cin + cout)
    x = NO.bits_f32(NO.bf16_bits(rng.normal(size=(nb, nz, ny, nx, cin)).astype(np.float32)))
    g = NO.bits_f32(NO.bf16_bits(rng.normal(size=(nb, nz, ny, nx, cout)).astype(np.float32)))
    dx, dg = bbpp.DeviceArray.from_host(NO.bf16_bits(x)), bbpp.DeviceArray.from_host(NO.bf16_bits(g))
    dW = bbpp.DeviceArray((27, cout, cin), np.float32)
    dW.zero()
    assert L.bbpp_conv3_wgrad(cin, cout, dx.ptr, cin, 0, dg.ptr, cout, dW.ptr, nx, ny, nz, nb, 1, 1, 0) == 0
    xp = np.pad(x.astype(np.float64), ((0, 0), (1, 1), (0, 0), (0, 0), (0, 0)))
    xp = np.pad(xp, ((0, 0), (0, 0), (1, 1), (1, 1), (0, 0)), mode="wrap")
    gf = g.astype(np.float64).reshape(-1, cout)
    want = np.empty((27, cout, cin))
    for t in range(27):
        dz, dy, dxx = t // 9, t // 3 % 3, t % 3
        want[t] = gf.T @ xp[:, dz:dz + nz, dy:dy + ny, dxx:dxx + nx].reshape(-1, cin)
    # FP32 sums of about 2e5 products of unit variance: 2^-24 sqrt(2 n) of a sum's
    # standard deviation sqrt(n) a rounding, over chains below 1000 steps
    n = nb * nx * ny * nz
    assert np.abs(dW.download() - want).max() <= 2.0 ** -24 * 1000 * np.sqrt(n)
