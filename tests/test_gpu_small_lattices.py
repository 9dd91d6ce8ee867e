"""GPU: the drop-in on D2Q9 lattices on both sides of the limits between its
small-lattice step kernels (9,728 and 48,640 cells of the linear range: one block of
two warps per SM, one-warp blocks, the large-lattice kernel), bit for bit
against the oracle with a Monitor on every second iteration.
"""
import pytest

from parity_util import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(20, 12), (120, 73), (120, 78), (121, 77), (160, 130), (160, 136), (250, 147), (250, 153), (255, 148), (300, 155), (300, 162)])
def test_small_lattices_match_oracle(built, nx, ny):
    import imexlb as im
    from oracle import orc
    args = dict(charlength=0.2 * ny / nx, xpos=0.3, re=40.0, ome=1.75, dt=1.0, rho0=1.0)
    cfg = im.make_config(2, nx, ny, **args)
    st = im.Setup(cfg)
    o = orc.Oracle(orc.make_input(2, nx, ny, **args))
    o.init_up(st.r_vec)
    o.init_pdf()
    with im.Solver(cfg) as s:
        s.set_geometry(st)
        s.upload(o.f, o.fb, o.p, o.u)
        assert s.fill_mode() == im.FILL_FUSED
        log = s.step(0, 21, 2)
        got = s.download()
    assert_same(log, o.run(0, 21, 2), "Monitor")
    for name, a, b in zip(("f", "fb", "p", "u"), got, (o.f, o.fb, o.p, o.u)):
        assert_same(a, b, name)
