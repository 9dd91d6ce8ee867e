"""CPU: the device's plane stride at the limit of 32-bit slots.

A lattice whose populations still have 32-bit slot indices (cells * Q <
2^31 - 1) must keep them, and every D2Q9 stride must be even: the kernels that
update two neighbouring cells per thread read and write words of two
elements, which start on an odd element of every other plane if it is not.
"""
import pytest

LIMIT = 2 ** 31 - 1


def _cells2(nx, ny):
    return (nx + 1 + 6) * (ny + 1 + 6)


@pytest.mark.parametrize("nx,ny", [(8112, 29382), (2852, 83452)])
def test_odd_lattices_at_the_limit(built, nx, ny):
    import imexlb as im
    n = _cells2(nx, ny)
    assert n % 2 == 1 and n * 9 < LIMIT <= -(-n // 64) * 64 * 9
    s = im.lib().imexlb_testing_plane_stride(n, 9)
    assert s % 2 == 0 and n <= s < n + 64 and s * 9 < LIMIT


@pytest.mark.parametrize("q", [9, 27])
def test_strides_around_the_limit(built, q):
    import imexlb as im
    last = (LIMIT - 1) // q  # the last number of cells with 32-bit slots
    for n in list(range(1, 200)) + list(range(last - 200, last + 200)) + list(range(2 ** 32 - 3, 2 ** 32 + 3)):
        s = im.lib().imexlb_testing_plane_stride(n, q)
        full = -(-n // 64) * 64
        assert n <= s <= full
        if n * q < LIMIT:
            assert s * q < LIMIT  # 32-bit slots are kept
            # no larger power of two up to 64 would do
            a = 64
            while a > 1 and -(-n // a) * a * q >= LIMIT:
                a //= 2
            assert s == -(-n // a) * a
        else:
            assert s == full
        if q == 9:
            assert s % 2 == 0
