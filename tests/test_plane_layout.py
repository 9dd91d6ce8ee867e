"""CPU: the device layout with aligned planes.

On the device every SoA plane takes NP elements, the padded cells N rounded up
to 64, and the linear cell range starts at id_lo rounded down to a multiple of 64,
so that a warp's 32 cells start on a 128-byte (4-byte storage) or 64-byte
(2-byte) boundary in every plane. Restated here with the host layout of every
lattice the tests and the benchmark run: the cells added below id_lo are ghost
cells (masked out), no pull of a fluid node leaves its buffer, and the staged
kernel's copies (TILE * 2 + 16 bytes from the 16-byte boundary below a run, the
mask's TILE + 16) stay inside the Q * NP elements and NP mask bytes.
"""
import numpy as np
import pytest

from test_staged_layout import GHOST, cases, fits, layout

ALIGN, TILE, ESZ = 64, 1024, 2


@pytest.mark.parametrize("case", cases(), ids=lambda c: c[0])
def test_aligned_planes(case):
    import imexlb as im
    name, dim, nx, ny, nz = case
    cfg = im.make_config(dim, nx, ny, nz)
    t, e = im.lattice(dim)
    Q = t.size
    N, id_lo, id_hi, dy, dz, off = layout(cfg, e)
    NP = -(-N // ALIGN) * ALIGN
    lo = id_lo // ALIGN * ALIGN
    assert 0 <= lo <= id_lo and id_lo - lo < ALIGN and N <= NP < N + ALIGN
    # the cells in [lo, id_lo) lie before the first interior node, hence ghosts
    first = GHOST + dy * GHOST + dz * GHOST
    assert id_lo == first
    for esz in (2, 4, 8):
        for q in range(Q):
            assert (esz * (q * NP + lo)) % (ALIGN * esz) == 0
            # the outermost fluid nodes' pulls
            for c in (id_lo, id_hi - 1):
                assert 0 <= q * NP + c - off[q] < Q * NP
    if not fits(N, id_hi, dy, dz, TILE):
        return
    run = TILE * ESZ + 16
    tiles = lo + TILE * np.arange((id_hi - lo + TILE - 1) // TILE, dtype=np.int64)
    for q in range(Q):
        a = ESZ * (q * NP - off[q] + tiles)
        a0 = a & ~np.int64(15)
        assert np.all(a0 >= 0) and np.all(a0 + run <= ESZ * Q * NP), (name, q)
        assert np.all(a + ESZ * (TILE + 1) <= a0 + run)
        assert np.all(a - a0 == a[0] - a0[0])
    m0 = tiles & ~np.int64(15)
    assert np.all(m0 >= 0) and np.all(m0 + TILE + 16 <= NP)
