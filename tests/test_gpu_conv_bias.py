"""GPU: a layer that stores fewer channels than its GEMM computes takes a
bias of as many values as it stores. The bias here ends a buffer whose next
values are NaN, first as one of the stored count, then with every channel's
value given: both must give the float64 reference within its rounding (the
bound of test_gpu_conv_tiles.py, one addition more)."""
import ctypes as C

import pytest

from test_gpu_conv_tiles import ULP, _conv64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("store", [1, 3, 16, 20])
def test_bias_of_the_stored_channels(built, store):
    import torch
    import imexlb as im
    from imexlb.neural import _p
    torch.manual_seed(store)
    L = im.lib()
    n, h, w, cin, cout = 2, 9, 17, 16, 32
    d = im.ConvDesc(n, h, w, cin, h, w, cout, store, 1, 0)
    x = torch.randn(n, h, w, cin, device="cuda").to(torch.bfloat16)
    wt = torch.randn(cout, 9 * cin, device="cuda").to(torch.bfloat16)
    buf = torch.full((64,), float("nan"), device="cuda")
    buf[:store] = torch.randn(store, device="cuda")
    full = torch.zeros(cout, device="cuda")
    full[:store] = buf[:store]
    y, yf = (torch.empty(n, h, w, store, device="cuda") for _ in range(2))
    assert L.imexlb_nn_conv_fwd(C.byref(d), _p(x), _p(wt), _p(buf), 0, None, _p(y), None) == 0
    assert L.imexlb_nn_conv_fwd(C.byref(d), _p(x), _p(wt), _p(full), 0, None, _p(yf), None) == 0
    assert torch.equal(y, yf)
    x6, w6, b6 = x.double(), wt.double(), buf[:store].double()
    ref = _conv64(x6, w6, 1, 0)[..., :store] + b6
    mag = _conv64(x6.abs(), w6.abs(), 1, 0)[..., :store] + b6.abs()
    assert bool(((y.double() - ref).abs() <= (9 * cin + 1) * ULP * mag).all())
