"""GPU: batches of more cases than one launch takes, with every kind of case.

The batched step runs the same explicitly rounded operations as the
single-case kernels, so a case must come out of a batch with the bits it has
when stepped alone: f, fb, p and u of every case, over several calls with
unequal budgets (runs replayed from graphs and single launches), for cases
whose boundary copies run inside the step and cases that keep the separate
list, in 2D and 3D, and across a switch to the persistent kernel.
"""
import numpy as np
import pytest

from parity_util import assert_same

pytestmark = pytest.mark.gpu


def _cfgs(im, dim, n):
    rng = np.random.default_rng(n)
    out = []
    for k in range(n):
        if dim == 2:
            nx, ny = int(rng.integers(30, 140)), int(rng.integers(20, 90))
            L = rng.uniform(0.1, 0.25) * ny / nx
            out.append(im.make_config(2, nx, ny, charlength=L, xpos=0.3, re=50.0, ome=1.7,
                                      yoff=float(rng.uniform(-2, 2))))
        else:
            nx, ny, nz = (int(v) for v in rng.integers(18, 40, 3))
            out.append(im.make_config(3, nx, ny, nz, charlength=0.3 * min(ny, nz) / nx, xpos=0.4, re=30.0,
                                      ome=1.6))
    return out


def _solver(im, cfg, prec, seed):
    st = im.Setup(cfg, seed=seed)
    if cfg.dim == 2 and seed % 5 == 4:
        # one more obstacle cell, one row inside the wall: no fused plan
        cell = (20 + 3) + cfg.dy * (1 + 3)
        assert st.geo[cell] == 1
        st.geo[cell] = 0
        st.fluid_id = st.fluid_id[st.fluid_id != cell]
        st.b_user = np.sort(np.append(st.b_user, cell)).astype(np.int32)
    s = im.Solver(cfg, precision=prec)
    s.set_geometry(st)
    s.init_state(st.r_vec)
    s.init_pdf()
    s.step(0, 1)
    return s


@pytest.mark.parametrize("dim,n,prec", [(2, 37, "FP32"), (2, 1, "FP16"), (2, 18, "BF16"), (3, 5, "FP32"),
                                        (3, 3, "FP16")])
def test_batch_bits(built, dim, n, prec):
    import imexlb as im
    code = getattr(im, prec)
    cfgs = _cfgs(im, dim, n)
    alone = [_solver(im, c, code, k) for k, c in enumerate(cfgs)]
    batched = [_solver(im, c, code, k) for k, c in enumerate(cfgs)]
    modes = {s.fill_mode() for s in batched}
    if dim == 2 and n > 4:
        assert modes == {im.FILL_FUSED, im.FILL_KERNEL}
    rng = np.random.default_rng(1)
    with im.Batch(batched) as b:
        for lo, hi in ((0, 4), (0, 40), (8, 9), (17, 18)):
            steps = rng.integers(lo, hi, n).astype(np.int32)
            b.step(steps=steps)
            for s, k in zip(alone, steps):
                s.step(1, int(k))
    for k, (s, a) in enumerate(zip(batched, alone)):
        for name, x, y in zip(("f", "fb", "p", "u"), s.download(), a.download()):
            assert_same(x, y, "case %d %s" % (k, name))


def test_modes_alternate(built):
    """Lockstep and persistent calls on the same cases, single steps between
    (the persistent kernel and a single step in the separate-list mode pull
    the ghost slots that lockstep's fused steps leave out)."""
    import imexlb as im
    cfgs = _cfgs(im, 2, 6)
    alone = [_solver(im, c, im.FP32, k) for k, c in enumerate(cfgs)]
    batched = [_solver(im, c, im.FP32, k) for k, c in enumerate(cfgs)]
    with im.Batch(batched) as b:
        for mode in (im.BATCH_LOCKSTEP, im.BATCH_PERSISTENT, im.BATCH_LOCKSTEP, im.BATCH_PERSISTENT):
            b.set_mode(mode)
            b.step(11)
            for s in batched:
                if s.fill_mode() == im.FILL_FUSED and mode == im.BATCH_LOCKSTEP:
                    s.set_fill_mode(im.FILL_KERNEL)
                s.step(1, 3)
                s.sample(16, 8)
    for s in alone:
        s.step(1, 4 * 14)
    for s, a in zip(batched, alone):
        for name, x, y in zip(("p", "u"), s.download()[2:], a.download()[2:]):
            # (test_gpu_batch_persistent's bound between the two kernels)
            fin = np.isfinite(y)
            assert np.array_equal(np.isfinite(x), fin), name
            assert np.abs(x[fin] - y[fin]).max() <= 2e-6 * np.abs(y[fin]).max(), name
