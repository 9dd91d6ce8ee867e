"""GPU: every launch shape that the tuner of a batch may choose, bit for bit.

On D2Q9 shapes 0, 1, 2 and 5 update one cell per thread (k_step_batch), shapes 3
and 4 and the single-lattice step two neighbouring ones (k_step_batch_pair,
k_step_pair) with word accesses: the sizes have odd and even row strides, an odd
number of cells, lattices of less than a block and obstacles in reach of the
walls and the inlet, with the boundary copies in the step and, for one more obstacle
cell beside a wall, in the separate list. All run the same explicitly rounded
operations, so populations, p and u must have the bits of the one-cell shape of
128 threads; the same for the six shapes in 3D and the single-lattice step
there.
"""
import ctypes as C

import numpy as np
import pytest

from parity_util import assert_same

pytestmark = pytest.mark.gpu


def _solver(im, dims, prec, separate):
    dim = len(dims)
    if dim == 2:
        nx, ny = dims
        cfg = im.make_config(2, nx, ny, charlength=0.4 * ny / nx, xpos=0.3, re=8.0, ome=1.6)
    else:
        cfg = im.make_config(3, *dims, charlength=0.35 * min(dims[1:]) / dims[0], xpos=0.4, re=20.0, ome=1.6)
    st = im.Setup(cfg, seed=4)
    if separate:
        # one row inside the wall: no fused plan
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


def _check(im, dims, prec, separate=False):
    code = getattr(im, prec)
    sol = [_solver(im, dims, code, separate) for _ in range(7)]
    assert (sol[0].fill_mode() == im.FILL_FUSED) == (not separate)
    for shape in range(6):
        with im.Batch([sol[shape]]) as b:
            assert im.lib().imexlb_testing_batch_shape(b.b, shape) == 0
            b.step(11)
            b.step(8)
    sol[6].step(1, 19)
    out = [s.download() for s in sol]
    for k in range(1, 7):
        for name, x, y in zip(("f", "fb", "p", "u"), out[k], out[0]):
            assert_same(x, y, "%s %s" % ("shape %d" % k if k < 6 else "single", name))
    for s in sol:
        s.close()


@pytest.mark.parametrize("prec", ["FP32", "FP16", "BF16"])
@pytest.mark.parametrize("dims", [(12, 8), (13, 8), (20, 13), (33, 17), (62, 31), (63, 32), (129, 66), (250, 5)])
def test_shapes_2d(built, dims, prec):
    import imexlb as im
    _check(im, dims, prec)


@pytest.mark.parametrize("prec,dims", [("FP32", (63, 32)), ("FP16", (62, 31)), ("BF16", (129, 66))])
def test_shapes_with_separate_boundary_list(built, prec, dims):
    import imexlb as im
    _check(im, dims, prec, separate=True)


@pytest.mark.parametrize("prec", ["FP32", "FP16", "BF16"])
@pytest.mark.parametrize("dims", [(14, 10, 9), (33, 16, 17)])
def test_shapes_3d(built, dims, prec):
    import imexlb as im
    _check(im, dims, prec)


def test_bad_shapes_are_refused(built):
    import imexlb as im
    s = _solver(im, (20, 13), im.FP32, False)
    with im.Batch([s]) as b:
        assert im.lib().imexlb_testing_batch_shape(b.b, -1) != 0
        assert im.lib().imexlb_testing_batch_shape(b.b, 6) != 0
    assert im.lib().imexlb_testing_batch_shape(C.c_void_p(), 0) != 0
    s.close()
