"""GPU: the forms of the fixed-point collision (the lattices' own weights with
1 - ome positive, zero and negative; any weights, taken where ome t_i is not
a multiple of 2^-63) against the double-precision oracle.

Bound: every population takes three roundings of at most 2^-61 per iteration
and the oracle's double about as much at |f| < 0.1, so 30 iterations with the sums over
27 directions stay below 30 * 27 * 2^-58 = 2.9e-15; a factor of 30 is left
for their growth through the flow.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("ome", [0.03, 0.1, 0.75, 1.0, 1.6, 1.95])
def test_fixed_point_forms_match_double(built, dim, ome):
    import imexlb as im
    from oracle import orc
    size = (61, 33) if dim == 2 else (33, 18, 19)
    nu = (1.0 / ome - 0.5) / 3.0
    # an inlet velocity of 0.03, inside the kind's range (0.25), whatever ome is
    args = dict(charlength=0.15, xpos=0.3, re=0.03 * 0.15 * size[0] / nu, ome=ome, dt=1.0, rho0=1.0)
    cfg = im.make_config(dim, *size, **args)
    st = im.Setup(cfg)
    o = orc.Oracle(orc.make_input(dim, *size, **args))
    o.init_up(st.r_vec)
    o.init_pdf()
    # populations of a developed magnitude
    o.f[:] = np.random.default_rng(3).uniform(-0.01, 0.01, o.f.size)
    with im.Solver(cfg, precision=im.FIX64) as s:
        s.set_geometry(st)
        s.upload(o.f, o.fb, o.p, o.u)
        s.step(0, 30, 10)
        f, _, p, u = s.download()
    o.run(0, 30, 10)
    assert np.all(np.isfinite(f))
    for a, b in ((f, o.f), (p, o.p), (u, o.u)):
        assert np.max(np.abs(a - b)) < 1e-13
