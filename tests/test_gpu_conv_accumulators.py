"""GPU: no weight-gradient accumulator takes more than 4096 output pixels.

The tensor cores accumulate in FP32 and truncate, so a long sum loses its small
terms. One pixel's product is 2^20, whose FP32 unit is 2^-3, and every other
pixel's 2^-10: the 16 pixels of an MMA add 2^-6, which that one accumulator drops
from then on. All other partial sums are exact (multiples of 2^-10 below 2^13),
and so is their sum in dw wherever they are multiples of 2^-3, which whole tiles
of 128 pixels are. The error of the centre tap is therefore at most 4096 * 2^-10 = 4;
accumulators of one block's share of the pixels, four times 4096 here, would lose
16.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,yblocks", [(16, 16, 1), (32, 48, 1), (64, 64, 2)])
def test_accumulators_are_bounded(built, cin, cout, yblocks):
    import torch
    import imexlb as im
    from imexlb.neural import _p
    L = im.lib()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 4 * 32 * sms // yblocks  # images of one 8 x 16 tile
    d = im.ConvDesc(n, 16, 8, cin, 16, 8, cout, 0, 1, 0)
    x = torch.ones(n, 16, 8, cin, dtype=torch.bfloat16, device="cuda")
    dz = torch.full((n, 16, 8, cout), 2.0 ** -10, dtype=torch.bfloat16, device="cuda")
    dz[0, 0, 0] = 2.0 ** 20
    dw = torch.zeros(cout, 9, cin, device="cuda")
    assert L.imexlb_nn_conv_bwd_weight(C.byref(d), _p(x), _p(dz), _p(dw), None) == 0
    exact = 2.0 ** 20 + (n * 128 - 1) * 2.0 ** -10
    err = (dw[:, 4].double() - exact).abs()
    assert float(err.max()) <= 4096 * 2.0 ** -10
    st = C.c_int(-1)
    assert L.imexlb_nn_status(C.byref(st)) == 0 and st.value == 0
