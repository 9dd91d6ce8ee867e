"""GPU: the data gradient with weights at every 2-byte offset of a 16-byte
boundary, which it has always taken: the same bits as with aligned weights,
and the aligned call leaves its scratch memory alone."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,stride,up", [(16, 64, 1, 0), (48, 48, 1, 1), (64, 16, 2, 0)])
def test_data_gradient_takes_any_weight_address(built, cin, cout, stride, up):
    import torch
    import imexlb as im
    from imexlb.neural import _p
    torch.manual_seed(cin)
    L = im.lib()
    n, h, w = 2, 13, 22
    hg, wg = (2 * h, 2 * w) if up else (h, w)
    d = im.ConvDesc(n, h, w, cin, (hg - 1) // stride + 1, (wg - 1) // stride + 1, cout, 0, stride, up)
    nw = 9 * cin * cout
    buf = torch.zeros(nw + 8, dtype=torch.bfloat16, device="cuda")
    wt = torch.randn(nw, device="cuda").to(torch.bfloat16)
    dz = torch.randn(n, d.hout, d.wout, cout, device="cuda").to(torch.bfloat16)

    def run(wp):
        dgrid = torch.full((n, hg, wg, cin), float("nan"), device="cuda")
        dx = torch.full((n, h, w, cin), float("nan"), device="cuda") if up else None
        scratch = torch.full((nw,), 7.0, dtype=torch.bfloat16, device="cuda")
        assert L.imexlb_nn_conv_bwd_data(C.byref(d), _p(dz), wp, _p(scratch), _p(dgrid), _p(dx), None) == 0
        return dgrid, dx, scratch

    assert buf.data_ptr() % 16 == 0 and wt.data_ptr() % 16 == 0
    ref, refx, scratch = run(_p(wt))
    assert bool(torch.isfinite(ref).all()) and bool((scratch == 7.0).all())
    for k in range(1, 8):
        buf.zero_()
        buf[k:k + nw] = wt
        got, gotx, _ = run(C.c_void_p(buf.data_ptr() + 2 * k))
        assert torch.equal(got, ref)
        if up:
            assert torch.equal(gotx, refx)
