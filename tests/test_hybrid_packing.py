"""Token lists of a step are packed as int() and numpy would pack them one by one: every form of list, and the same refusals."""
import numpy as np
import pytest

from jacobiforcing_b200.hybrid_runtime import _packed


def test_packing_equals_one_by_one():
    parts = [[1, 2, 3], (4,), np.arange(5, dtype=np.int64), np.array([7.9, 8.0]), [np.int32(9), np.uint8(255)], range(3), iter([6, 5]), [True, 2.5],
             [], np.array([], dtype=np.int32), ["12"], np.arange(10)[::-3], b"ab"]
    again = [[6, 5] if hasattr(p, "__next__") else p for p in parts]
    got, start = _packed(parts)
    want = [int(x) for p in again for x in p]
    assert got.dtype == np.int32 and got.tolist() == want
    assert start == [0] + np.cumsum([len(p) for p in again]).tolist()


def test_no_lists_and_empty_lists():
    got, start = _packed([])
    assert got.dtype == np.int32 and len(got) == 0 and start == [0]
    got, start = _packed([[], ()])
    assert len(got) == 0 and start == [0, 0, 0]


@pytest.mark.parametrize("bad,err", [([2 ** 31], OverflowError), ([-2 ** 31 - 1], OverflowError), (np.array([2 ** 40]), OverflowError), ([float("nan")], ValueError),
                                     ([None], TypeError), (["x"], ValueError)])
def test_refusals(bad, err):
    with pytest.raises(err):
        _packed([[1], bad])


@pytest.mark.filterwarnings("ignore::DeprecationWarning")
def test_arrays_whose_rows_are_single_numbers():
    for column in (np.array([[5], [6]]), np.array([[[7]]]), [np.array([4])]):
        got, start = _packed([column, [1]])
        assert got.tolist() == [int(x) for x in column] + [1] and start == [0, len(column), len(column) + 1]
