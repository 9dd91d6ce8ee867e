"""CPU: how a batch is divided into launches. A part is one launch an
iteration, so small cases must share few of them: a batch that fits one part's
room is one part, whatever its cases' sizes, and many small cases need no more
parts than their bytes and the launch's 128 cases ask for."""
import ctypes as C

import numpy as np
import pytest

ROOM = 31 << 20
CAP = 128


def _plan(sizes):
    import imexlb as im
    b = np.ascontiguousarray(sizes, dtype=np.int64)
    part, chain = (np.full(b.size, -1, dtype=np.int32) for _ in range(2))
    n = im.lib().imexlb_testing_batch_plan(b.ctypes.data_as(C.POINTER(C.c_longlong)), b.size, ROOM,
                                           part.ctypes.data_as(C.POINTER(C.c_int)),
                                           chain.ctypes.data_as(C.POINTER(C.c_int)))
    assert n > 0 and set(part) == set(range(n))
    for k in range(n):
        assert len(set(chain[part == k])) == 1
    return n, part, chain, b


@pytest.mark.parametrize("n", [1, 2, 3, 8, 17, 64, 100, 128])
def test_what_fits_is_one_part(built, n):
    sizes = np.random.default_rng(n).integers(100_000, 240_000, n)
    assert _plan(sizes)[0] == 1


@pytest.mark.parametrize("n", [129, 300, 1000])
def test_many_small_cases(built, n):
    sizes = np.random.default_rng(n).integers(100_000, 400_000, n)
    parts, part, _, b = _plan(sizes)
    assert max(np.bincount(part)) <= CAP and max(np.bincount(part, b)) <= ROOM
    # first fit, largest first: at most 11/9 of the fewest, and one
    assert parts <= 11 / 9 * max(-(-n // CAP), -(-int(b.sum()) // ROOM)) + 1


def test_two_parts_are_alike(built):
    parts, part, chain, b = _plan([520_000] * 64)  # 63 of them would fit
    assert parts == 2 and list(np.bincount(part)) == [32, 32] and set(chain) == {0, 1}
    parts, part, _, b = _plan(np.linspace(100_000, 500_000, 150))
    used = np.bincount(part, b)
    assert parts == 2 and abs(used[0] - used[1]) <= b.max()


def test_large_cases_are_parts_of_their_own(built):
    parts, part, chain, b = _plan([3 * ROOM, ROOM + 1, ROOM + 1, ROOM, 5, 5])
    assert parts == 5
    for i in range(4):
        assert np.count_nonzero(part == part[i]) == 1
    assert part[4] == part[5]
    load = np.bincount(chain, b)
    assert abs(load[0] - load[1]) <= b[1] + 10
