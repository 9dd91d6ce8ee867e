"""GPU: the D2Q9 step that updates two neighbouring cells per thread, where its
word accesses can go wrong: odd and even row strides, an odd number of
cells, lattices of a few blocks, obstacles in reach of the walls and the
inlet. The batched step updates one cell per thread with the same explicitly
rounded operations, so every population, p and u must have its bits; the
next Monitor value is the largest speed of the downloaded u, within the rounding
of three float operations (3 * 2^-24).
"""
import numpy as np
import pytest

from parity_util import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["FP32", "FP16", "BF16"])
@pytest.mark.parametrize("nx,ny", [(12, 8), (13, 8), (20, 13), (33, 17), (62, 31), (63, 32), (129, 66), (250, 5)])
def test_pairs_match_single_cells(built, nx, ny, prec):
    import imexlb as im
    cfg = im.make_config(2, nx, ny, charlength=0.4 * ny / nx, xpos=0.3, re=8.0, ome=1.6)
    sol = []
    for _ in range(2):
        st = im.Setup(cfg, seed=4)
        s = im.Solver(cfg, precision=getattr(im, prec))
        s.set_geometry(st)
        s.init_state(st.r_vec)
        s.init_pdf()
        s.step(0, 1)
        sol.append(s)
    one, ref = sol
    one.step(1, 11)
    with im.Batch([ref]) as b:
        b.step(11)
    got, want = one.download(), ref.download()
    log = one.step(12, 1, 12)  # Monitor comes before the iteration's collision
    for name, x, y in zip(("f", "fb", "p", "u"), got, want):
        fin = np.isfinite(y)
        assert np.array_equal(np.isfinite(x), fin)
        assert_same(np.asarray(x)[fin], np.asarray(y)[fin], name)
    ids = np.asarray(st.fluid_id)[1:]
    u = np.asarray(got[3]).reshape(-1, 2)[ids]
    umax = np.sqrt((u.astype(np.float64) ** 2).sum(1)).max()
    assert log.size == 1 and abs(float(log.ravel()[-1]) - umax) <= 3 * 2.0 ** -24 * umax
    for s in sol:
        s.close()
