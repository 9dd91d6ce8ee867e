"""GPU: the network's kernels start while the previous kernel of their stream
ends, and must still see all it wrote: a chain of parameter update, forward
convolution, ReLU gradient, weight gradient and data gradient without a
synchronisation gives the bits of the same chain with one after every call
(dW and the bias gradient, summed by atomics in any order, within
2^-24 sqrt(terms) of their largest value times 8), also replayed from a
captured graph.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,cin,cout,stride,up", [(1, 16, 24, 16, 48, 1, 0), (3, 33, 41, 48, 48, 1, 1),
                                                      (2, 37, 50, 64, 32, 2, 0)])
def test_chain_without_synchronisation(built, n, h, w, cin, cout, stride, up):
    torch = pytest.importorskip("torch")
    import imexlb as im
    L = im.lib()
    hg, wg = (2 * h, 2 * w) if up else (h, w)
    ho, wo = (hg - 1) // stride + 1, (wg - 1) // stride + 1
    d = im.ConvDesc(n, h, w, cin, ho, wo, cout, 0, stride, up)
    g = torch.Generator(device="cuda").manual_seed(2)

    def rnd(*s):
        return torch.randn(s, device="cuda", generator=g)

    x, dy = rnd(n, h, w, cin).bfloat16(), rnd(n, ho, wo, cout)
    p0, grad, bias = rnd(cout, 9 * cin) * 0.1, rnd(cout, 9 * cin), rnd(cout) * 0.1
    wt = torch.empty(cin, 9 * cout, dtype=torch.bfloat16, device="cuda")

    def buffers():
        return dict(p=p0.clone(), m=torch.zeros_like(p0), v=torch.zeros_like(p0), pb=torch.zeros_like(p0).bfloat16(),
                    y=torch.zeros(n, ho, wo, cout, dtype=torch.bfloat16, device="cuda"),
                    dz=torch.zeros(n, ho, wo, cout, dtype=torch.bfloat16, device="cuda"),
                    db=torch.zeros(cout, device="cuda"), dw=torch.zeros(cout, 9 * cin, device="cuda"),
                    dg=torch.zeros(n, hg, wg, cin, device="cuda"),
                    dx=torch.zeros(n, h, w, cin, device="cuda") if up else None)

    def ptr(t):
        return C.c_void_p(t.data_ptr()) if t is not None else None

    def chain(b, stream, after):
        s = C.c_void_p(stream.cuda_stream)
        b["db"].zero_()
        b["dw"].zero_()
        for call in (
                lambda: L.imexlb_nn_adam(ptr(b["p"]), ptr(grad), ptr(b["m"]), ptr(b["v"]), ptr(b["pb"]), p0.numel(),
                                         0.05, 0.9, 0.999, 1e-8, 1, 0.0, s),
                lambda: L.imexlb_nn_conv_fwd(C.byref(d), ptr(x), ptr(b["pb"]), ptr(bias), 1, ptr(b["y"]), None, s),
                lambda: L.imexlb_nn_act_grad(ptr(dy), ptr(b["y"]), dy.numel(), cout, 1, ptr(b["dz"]), ptr(b["db"]), s),
                lambda: L.imexlb_nn_conv_bwd_weight(C.byref(d), ptr(x), ptr(b["dz"]), ptr(b["dw"]), s),
                lambda: L.imexlb_nn_conv_bwd_data(C.byref(d), ptr(b["dz"]), ptr(b["pb"]), ptr(wt), ptr(b["dg"]),
                                                  ptr(b["dx"]), s)):
            assert call() == 0
            after()

    def same(a, b):
        for k in ("p", "pb", "y", "dz", "dg") + (("dx",) if up else ()):
            assert torch.equal(a[k], b[k]), k
        terms = n * ho * wo
        for k in ("db", "dw"):
            tol = 8 * 2.0 ** -24 * np.sqrt(terms) * float(a[k].abs().max())
            assert float((a[k] - b[k]).abs().max()) <= tol, k

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ref = buffers()
        chain(ref, stream, stream.synchronize)
        for _ in range(3):
            got = buffers()
            chain(got, stream, lambda: None)
            stream.synchronize()
            same(ref, got)
        rep = buffers()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            chain(rep, torch.cuda.current_stream(), lambda: None)
        for _ in range(2):
            rep["p"].copy_(p0)
            rep["m"].zero_()
            rep["v"].zero_()
            graph.replay()
            stream.synchronize()
            same(ref, rep)
    st = C.c_int(-1)
    assert L.imexlb_nn_status(C.byref(st)) == 0 and st.value == 0
