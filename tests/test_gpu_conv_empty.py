"""GPU: layers without pixels. A forward pass of nothing succeeds and writes
nothing; a weight gradient of nothing is refused (-2) and leaves dw as it was,
like the data gradient of an upsampled layer, which has no sums to form."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(0, 8), (8, 0), (0, 0)])
def test_no_pixels(built, h, w):
    import torch
    import imexlb as im
    from imexlb.neural import _p
    L = im.lib()
    x = torch.randn(16 * 64, device="cuda").to(torch.bfloat16)
    wt = torch.randn(16 * 9 * 16, device="cuda").to(torch.bfloat16)
    for up in (0, 1):
        d = im.ConvDesc(1, h, w, 16, h << up, w << up, 16, 0, 1, up)
        out = torch.full((4096,), 3.0, device="cuda")
        dx = torch.full((4096,), 3.0, device="cuda")
        dw = torch.randn(16, 9 * 16, device="cuda")
        keep = dw.clone()
        assert L.imexlb_nn_conv_fwd(C.byref(d), _p(x), _p(wt), None, 0, None, _p(out), None) == 0
        assert L.imexlb_nn_conv_bwd_weight(C.byref(d), _p(x), _p(x), _p(dw), None) == -2
        rc = L.imexlb_nn_conv_bwd_data(C.byref(d), _p(x), _p(wt), _p(wt), _p(out), _p(dx), None)
        assert rc == (-2 if up else 0)
        torch.cuda.synchronize()
        assert torch.equal(dw, keep)
        assert bool((out == 3.0).all()) and bool((dx == 3.0).all())
    st = C.c_int(-1)
    assert L.imexlb_nn_status(C.byref(st)) == 0 and st.value == 0
