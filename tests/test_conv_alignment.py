"""CPU: the checks on the convolutions' arguments. Their kernels copy x, w and dz 16
bytes at a time, so a pointer off that boundary is refused before anything
touches the device (the addresses here are made up and are never read). The
data gradient's w is the exception: it may lie anywhere a bfloat16 may, if the
scratch memory is aligned (tests/test_gpu_conv_alignment.py)."""
import ctypes as C

import pytest

GOOD = 1 << 20


@pytest.mark.parametrize("off", [1, 2, 4, 8, 14])
def test_misaligned_inputs_are_refused(built, off):
    import imexlb as im
    L = im.lib()
    d = im.ConvDesc(1, 8, 8, 16, 8, 8, 16, 0, 1, 0)
    ok, bad = C.c_void_p(GOOD), C.c_void_p(GOOD + off)
    for x, w in ((bad, ok), (ok, bad), (bad, bad)):
        assert L.imexlb_nn_conv_fwd(C.byref(d), x, w, None, 0, ok, None, None) == -1
    assert L.imexlb_nn_conv_bwd_data(C.byref(d), bad, ok, ok, ok, None, None) == -1
    assert L.imexlb_nn_conv_bwd_data(C.byref(d), ok, bad, bad, ok, None, None) == -1
    for x, dz in ((bad, ok), (ok, bad), (bad, bad)):
        assert L.imexlb_nn_conv_bwd_weight(C.byref(d), x, dz, ok, None) == -1


def test_odd_weight_address_is_refused(built):
    import imexlb as im
    d = im.ConvDesc(1, 8, 8, 16, 8, 8, 16, 0, 1, 0)
    ok = C.c_void_p(GOOD)
    assert im.lib().imexlb_nn_conv_bwd_data(C.byref(d), ok, C.c_void_p(GOOD + 1), ok, ok, None, None) == -1


@pytest.mark.parametrize("h,w", [(-40, -40), (-1, 8), (8, -1), (-16, 0)])
def test_negative_sizes_are_refused(built, h, w):
    """(Their halo bounds would wrap around as unsigned numbers.)"""
    import imexlb as im
    L = im.lib()
    ok = C.c_void_p(GOOD)
    d = im.ConvDesc(1, h, w, 16, h, w, 16, 0, 1, 0)
    assert L.imexlb_nn_conv_fwd(C.byref(d), ok, ok, None, 0, ok, None, None) == -1
    assert L.imexlb_nn_conv_bwd_data(C.byref(d), ok, ok, ok, ok, None, None) == -1
    assert L.imexlb_nn_conv_bwd_weight(C.byref(d), ok, ok, ok, None) == -1
