"""GPU: the force sum at sizes on both sides of its one-block limit (1024
links) and with several links per thread, and downloads that leave fields out.

Both force sums are double-double, so they agree to one rounding of the
final value per component (the tolerance of test_gpu_observe: 4.5e-16 of the
summed magnitudes).
"""
import numpy as np
import pytest

from parity_util import assert_same

pytestmark = pytest.mark.gpu

CASES = [  # dim, nx, ny, nz, diameter / nx
    (2, 60, 40, 0, 0.02),     # a handful of links
    (2, 400, 300, 0, 0.5),    # 2D past one block
    (3, 40, 32, 32, 0.4),     # tens of blocks
    (3, 120, 84, 84, 0.6),    # several links per thread of every block
]


def _case(im, dim, nx, ny, nz, L):
    from oracle import orc
    args = dict(charlength=L, xpos=0.4, re=20.0, ome=1.7, dt=1.0, rho0=1.0)
    cfg = im.make_config(dim, nx, ny, nz, **args)
    st = im.Setup(cfg)
    o = orc.Oracle(orc.make_input(dim, nx, ny, nz, **args))
    o.init_up(st.r_vec)
    o.init_pdf()
    return cfg, st, o


@pytest.mark.parametrize("dim,nx,ny,nz,L", CASES)
def test_force_sum_sizes(built, dim, nx, ny, nz, L):
    import imexlb as im
    cfg, st, o = _case(im, dim, nx, ny, nz, L)
    with im.Solver(cfg) as s:
        s.set_geometry(st)
        s.upload(o.f, o.fb, o.p, o.u)
        for it in range(3):  # repeated samples reuse the counter
            _, F = s.step_observed(it, 1, 0, 1)
            o.run(it, 1, 0)
            Fo, n = o.forces()
            assert s.info().n_links == n > 0
            scale = 2 * np.abs(o.fb.reshape(-1, o.s.nq)[o.lists["fluid_id"]]).sum()
            assert np.all(np.abs(F[0] - Fo) <= 4.5e-16 * scale), (F[0], Fo)
            assert np.array_equal(s.observe()[0], F[0])


@pytest.mark.parametrize("prec", ["FP64", "FP16"])
def test_partial_downloads(built, prec):
    import imexlb as im
    cfg, st, o = _case(im, 3, 30, 20, 22, 0.3)
    with im.Solver(cfg, precision=getattr(im, prec)) as s:
        s.set_geometry(st)
        s.init_state(st.r_vec)
        s.init_pdf()
        fresh = s.download()
        assert_same(fresh[0], o.f, "f = feq on the device")
        assert_same(fresh[3], o.u, "InitUP")
        s.step(0, 4)
        _, _, p, u = s.download(f=False, fb=False)
        full = s.download()
        assert_same(p, full[2], "p")
        assert_same(u, full[3], "u")
        assert_same(s.download(fb=False, p=False, u=False)[0], full[0], "f")
        if prec == "FP64":
            o.run(0, 4, 0)
            for name, a, b in zip(("f", "fb", "p", "u"), full, (o.f, o.fb, o.p, o.u)):
                assert_same(a, b, name)
