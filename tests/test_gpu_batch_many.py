"""GPU: batches of more small cases than one launch takes, and of as many as it
takes (the last case's arguments end the launch's 32 KB of parameters). Every
case must have the bits that it has when stepped alone, with budgets that
differ from case to case. 16 cases and 17 are the two sides of the smaller
set of parameters."""
import numpy as np
import pytest

from parity_util import assert_same

pytestmark = pytest.mark.gpu


def _solvers(im, n, dim, prec):
    out = []
    for k in range(n):
        if dim == 2:
            nx, ny = 24 + 3 * (k % 11), 18 + 5 * (k % 3)
            cfg = im.make_config(2, nx, ny, charlength=0.2 * ny / nx, xpos=0.3, re=20.0, ome=1.6)
        else:
            cfg = im.make_config(3, 14 + k % 5, 10, 9, charlength=0.2, xpos=0.4, re=20.0, ome=1.5)
        st = im.Setup(cfg, seed=k % 7)
        s = im.Solver(cfg, precision=prec)
        s.set_geometry(st)
        s.init_state(st.r_vec)
        s.init_pdf()
        s.step(0, 1)
        out.append(s)
    return out


@pytest.mark.parametrize("n,dim,prec", [(16, 2, "BF16"), (17, 2, "FP16"), (16, 3, "FP32"), (17, 3, "FP32"),
                                        (127, 2, "FP16"), (128, 2, "FP32"), (129, 2, "BF16"), (270, 2, "FP32"),
                                        (128, 3, "FP32")])
def test_many_cases(built, n, dim, prec):
    import imexlb as im
    alone, batched = (_solvers(im, n, dim, getattr(im, prec)) for _ in range(2))
    rng = np.random.default_rng(n)
    with im.Batch(batched) as b:
        for lo, hi in ((0, 4), (5, 45)):
            steps = rng.integers(lo, hi, n).astype(np.int32)
            b.step(steps=steps)
            for s, k in zip(alone, steps):
                s.step(1, int(k))
    for k, (s, a) in enumerate(zip(batched, alone)):
        for name, x, y in zip(("f", "fb", "p", "u"), s.download(), a.download()):
            assert_same(x, y, "case %d %s" % (k, name))
    for s in alone + batched:
        s.close()
