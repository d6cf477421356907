"""Commit lists are packed as numpy by itself packs them: every form of list, and the same refusals."""
import numpy as np
import pytest

from jacobiforcing_b200.runtime import _triples


def by_numpy(x):
    return np.ascontiguousarray(np.asarray(x, dtype=np.int32)).reshape(-1, 3)


@pytest.mark.parametrize("x", [[], (), [(1, 2, 3)], [(i, 0, i) for i in range(100)], ((1, 2, 3), (4, 5, 6)), [[1, 2, 3], [4, 5, 6]], [(1, 2, 3), [4, 5, 6]], [[1, 2, 3], (4, 5, 6)],
                               [(1.9, 2, 3)], [(np.int64(1), np.uint8(2), True)], [(np.array(1), 2, 3)], np.arange(12).reshape(4, 3), np.arange(6), [1, 2, 3], (1, 2, 3),
                               [(1, 2, 3, 4, 5, 6), (7, 8, 9, 10, 11, 12)], [(1, 2), (3, 4), (5, 6)], [(1, 2, 3), np.array([4, 5, 6])], [((1, 2, 3),), ((4, 5, 6),)]], ids=repr)
def test_what_numpy_takes(x):
    got, want = _triples(x), by_numpy(x)
    assert got.dtype == want.dtype and got.shape == want.shape and got.tolist() == want.tolist() and got.flags.c_contiguous


@pytest.mark.parametrize("x", [[(1, 2), (3, 4, 5, 6)], [(1, 2, 3), (4, 5)], [(1,), (2, 3, 4), (5, 6)], [(1, 2, 3), {4, 5, 6}], [(1, 2, 3), {4: 0, 5: 0, 6: 0}], [(1, 2, 3), b"abc"],
                               [(1, 2, 3), range(2)], [(1, 2, None)], [(1, 2, (3, 4))], [(1, 2, 2 ** 31)], [(1, 2, 3), ()], [(1, 2), (3, 4)], {(1, 2, 3)}], ids=repr)
def test_what_numpy_refuses(x):
    with pytest.raises(Exception) as want:
        by_numpy(x)
    with pytest.raises(want.type):
        _triples(x)
