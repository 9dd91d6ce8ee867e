"""GPU: the ReLU / bias gradient and the squared-error kernels on both of
their paths (eight or four channels a thread; one value a thread for other
channel counts and alignments), against float64 torch.

dz is one rounding of an exact selection: equal bit for bit. A sum of n FP32
values is within n * 2^-24 of the sum of their magnitudes in any order.
"""
import pytest

pytestmark = pytest.mark.gpu

ULP2 = 2.0 ** -24


@pytest.mark.parametrize("npix,c,relu,shift", [
    (1, 8, 1, 0), (997, 48, 1, 0), (40000, 48, 0, 0), (513, 64, 1, 0), (300, 16, 1, 0), (77, 56, 1, 0),
    (501, 12, 1, 0), (333, 48, 1, 1)])
def test_act_grad(built, npix, c, relu, shift):
    import torch
    import imexlb as im
    from imexlb.neural import _p
    torch.manual_seed(npix)
    n = npix * c
    dy = torch.randn(n + shift, device="cuda")[shift:]
    y = torch.relu(torch.randn(n + shift, device="cuda")).to(torch.bfloat16)[shift:]
    dz = torch.empty(n + shift, dtype=torch.bfloat16, device="cuda")[shift:]
    db = torch.full((c,), 0.5, device="cuda")
    assert im.lib().imexlb_nn_act_grad(_p(dy), _p(y) if relu else None, n, c, relu, _p(dz), _p(db), None) == 0
    ref = torch.where(y.float() > 0, dy, torch.zeros_like(dy)) if relu else dy
    assert torch.equal(dz, ref.to(torch.bfloat16))
    r = ref.double().view(npix, c)
    assert bool(((db.double() - 0.5 - r.sum(0)).abs() <= (npix + 2) * ULP2 * (r.abs().sum(0) + 1)).all())


@pytest.mark.parametrize("npix,c,used,weighted,shift", [
    (1, 4, 3, False, 0), (1000, 16, 3, False, 0), (70001, 16, 3, True, 0), (513, 8, 6, True, 0),
    (129, 7, 3, False, 0), (300, 16, 16, False, 1)])
def test_mse(built, npix, c, used, weighted, shift):
    import torch
    import imexlb as im
    from imexlb.neural import _p
    torch.manual_seed(npix)
    y = torch.randn(npix * c + shift, device="cuda")[shift:].view(npix, c)
    t = torch.randn(npix, used, device="cuda")
    w = torch.rand(npix, device="cuda") if weighted else None
    dy = torch.full((npix * c + shift,), 7.0, device="cuda")[shift:].view(npix, c)
    loss = torch.zeros(1, device="cuda")
    assert im.lib().imexlb_nn_mse(_p(y), _p(t), _p(w), npix, c, used, _p(dy), _p(loss), None) == 0
    d = (y[:, :used] - t).double()  # (the kernel's subtraction, rounded once)
    wt = w.double()[:, None] if weighted else 1.0
    ref = torch.zeros(npix, c, dtype=torch.float64, device="cuda")
    ref[:, :used] = 2 * wt * d / (npix * used)
    assert bool(((dy.double() - ref).abs() <= 8 * ULP2 * ref.abs()).all())
    assert bool((dy[:, used:] == 0).all())
    want = float((wt * d * d).sum() / (npix * used))
    assert abs(float(loss) - want) <= (npix * used + 8) * ULP2 * want
