"""GPU: the tiled convolution kernels (8 x 16 output pixels, staged halos) at
the sizes where a tile, a channel group or a store path ends.

Reference: torch convolutions in float64 on the same bf16 values. Products of
two bf16 values are exact in FP32, so a K-term sum accumulated in FP32 (each
addition off by at most one unit in the last place, 2^-23, tensor cores
truncating included) is within K * 2^-23 of the sum of the products'
magnitudes; that bound, element by element, is the tolerance.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -23


def _conv64(x, w, stride, up):
    import torch.nn.functional as F
    cin, cout = x.shape[-1], w.shape[0]
    x = x.permute(0, 3, 1, 2)
    if up:
        x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
    w = w.reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
    return F.conv2d(x, w, stride=stride, padding=1).permute(0, 2, 3, 1)


def _grads64(x, w, dz, stride, up):
    """dgrid, dx, dw of _conv64."""
    g = x.repeat_interleave(2, 1).repeat_interleave(2, 2) if up else x
    g, w = g.clone().requires_grad_(True), w.clone().requires_grad_(True)
    _conv64(g, w, stride, 0).backward(dz)
    n, h, wd, c = x.shape
    dx = g.grad.view(n, h, 2, wd, 2, c).sum((2, 4)) if up else g.grad
    return g.grad, dx, w.grad


def _within(got, ref, mag, terms):
    err = (got.double() - ref).abs()
    assert bool((err <= terms * ULP * mag + 1e-30).all()), float((err / (terms * ULP * mag + 1e-30)).max())


SHAPES = [  # n, h, w, cin, cout, stride, upsample
    (1, 16, 8, 16, 16, 1, 0),    # one whole tile
    (2, 17, 9, 48, 48, 1, 0),    # one pixel into the next tile both ways
    (1, 15, 7, 64, 64, 1, 0),    # one short of it, the most channels (taps in two blocks)
    (1, 1, 1, 32, 48, 1, 0),     # a single pixel
    (2, 33, 18, 48, 32, 2, 0),   # stride 2 from odd and even sizes: every parity class
    (1, 2, 3, 16, 64, 2, 0),
    (3, 8, 5, 48, 16, 1, 1),     # upsampled, ragged
    (1, 9, 12, 32, 32, 2, 1),    # upsampled and strided: sums between parity classes
    (40, 16, 24, 16, 48, 1, 0),  # several tiles per block
]


@pytest.mark.parametrize("n,h,w,cin,cout,stride,up", SHAPES)
def test_layer_against_float64(built, n, h, w, cin, cout, stride, up):
    import torch
    import imexlb as im
    from imexlb.neural import _p
    torch.manual_seed(n * 1000 + h)
    L = im.lib()
    hg, wg = (2 * h, 2 * w) if up else (h, w)
    d = im.ConvDesc(n, h, w, cin, (hg - 1) // stride + 1, (wg - 1) // stride + 1, cout, 0, stride, up)
    x = torch.randn(n, h, w, cin, device="cuda").to(torch.bfloat16)
    wt = torch.randn(cout, 9 * cin, device="cuda").to(torch.bfloat16)
    dz = torch.randn(n, d.hout, d.wout, cout, device="cuda").to(torch.bfloat16)
    y = torch.empty(n, d.hout, d.wout, cout, device="cuda")
    dgrid = torch.empty(n, hg, wg, cin, device="cuda")
    dx = torch.empty(n, h, w, cin, device="cuda") if up else None
    dw = torch.zeros(cout, 9 * cin, device="cuda")
    scratch = torch.empty(cin, 9 * cout, dtype=torch.bfloat16, device="cuda")
    assert L.imexlb_nn_conv_fwd(C.byref(d), _p(x), _p(wt), None, 0, None, _p(y), None) == 0
    assert L.imexlb_nn_conv_bwd_data(C.byref(d), _p(dz), _p(wt), _p(scratch), _p(dgrid), _p(dx), None) == 0
    assert L.imexlb_nn_conv_bwd_weight(C.byref(d), _p(x), _p(dz), _p(dw), None) == 0
    x6, w6, z6 = x.double(), wt.double(), dz.double()
    _within(y, _conv64(x6, w6, stride, up), _conv64(x6.abs(), w6.abs(), stride, up), 9 * cin)
    ref, mag = _grads64(x6, w6, z6, stride, up), _grads64(x6.abs(), w6.abs(), z6.abs(), stride, up)
    _within(dgrid, ref[0], mag[0], 9 * cout)
    if up:
        _within(dx, ref[1], mag[1], 9 * cout + 4)
    _within(dw, ref[2], mag[2], n * d.hout * d.wout)
    st = C.c_int(-1)
    assert L.imexlb_nn_status(C.byref(st)) == 0 and st.value == 0


def test_store_paths_and_wide_inputs(built):
    """Fewer stored channels, an output that is not 32-byte aligned (both
    element by element) and more than 64 input channels."""
    import torch
    import imexlb as im
    from imexlb.neural import _p
    torch.manual_seed(5)
    L = im.lib()
    n, h, w, cin, cout = 2, 11, 19, 80, 16
    x = torch.randn(n, h, w, cin, device="cuda").to(torch.bfloat16)
    wt = torch.randn(cout, 9 * cin, device="cuda").to(torch.bfloat16)
    x6, w6 = x.double(), wt.double()
    ref, mag = _conv64(x6, w6, 1, 0), _conv64(x6.abs(), w6.abs(), 1, 0)
    for store, shift in ((3, 0), (16, 1), (16, 0)):
        d = im.ConvDesc(n, h, w, cin, h, w, cout, store, 1, 0)
        buf = torch.empty(n * h * w * store + shift, device="cuda")
        y = buf[shift:].view(n, h, w, store)
        assert L.imexlb_nn_conv_fwd(C.byref(d), _p(x), _p(wt), None, 0, None, _p(y), None) == 0
        _within(y, ref[..., :store], mag[..., :store], 9 * cin)
    d = im.ConvDesc(n, h, w, cin, h, w, cout, 0, 1, 0)
    dz = torch.randn(n, h, w, cout, device="cuda").to(torch.bfloat16)
    dw = torch.zeros(cout, 9 * cin, device="cuda")
    assert L.imexlb_nn_conv_bwd_weight(C.byref(d), _p(x), _p(dz), _p(dw), None) == 0
    _within(dw, _grads64(x6, w6, dz.double(), 1, 0)[2],
            _grads64(x6.abs(), w6.abs(), dz.double().abs(), 1, 0)[2], n * h * w)
    # 96 input channels: weights and rows past a block's shared memory
    d = im.ConvDesc(n, h, w, 96, h, w, cout, 0, 1, 0)
    x = torch.zeros(n, h, w, 96, dtype=torch.bfloat16, device="cuda")
    wt = torch.zeros(cout, 9 * 96, dtype=torch.bfloat16, device="cuda")
    y = torch.empty(n, h, w, cout, device="cuda")
    assert L.imexlb_nn_conv_fwd(C.byref(d), _p(x), _p(wt), None, 0, None, _p(y), None) == -2
