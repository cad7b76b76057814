"""A step's token ids in any container, checked against the vocabulary."""
import numpy as np
import pytest
import torch

from foundry_b200.engine.context import _token_ids


class Unwalked(np.ndarray):
    """An array that nobody may walk through id by id."""

    def __iter__(self):
        raise AssertionError("walked")


@pytest.mark.parametrize("dtype", [np.int64, np.int32, np.uint16, np.uint64])
def test_arrays_are_checked_as_a_whole(dtype):
    ids = np.array([5, 0, 99, 7], dtype=dtype).view(Unwalked)
    got = _token_ids(ids, 100)
    assert got.dtype == np.int64 and got.tolist() == [5, 0, 99, 7]
    assert _token_ids(ids[::2], 100).tolist() == [5, 99]


@pytest.mark.parametrize("tokens", [[5, 7], (5, 7), range(5, 8, 2), np.array([5, 7]), np.array([5.0, 7.9]),
                                    torch.tensor([5, 7]), torch.tensor([5.0, 7.0]), [5.0, 7.5],
                                    [np.int32(5), torch.tensor(7)], np.array([5, 7], dtype=object)])
def test_containers(tokens):
    got = _token_ids(tokens, 8)
    assert got.dtype == np.int64 and got.tolist() == [5, 7]
    with pytest.raises(ValueError, match="outside the vocabulary of 7"):
        _token_ids(tokens, 7)


@pytest.mark.parametrize("bad", [-1, 100, 2 ** 40, 2 ** 63, 2 ** 70])
@pytest.mark.parametrize("make", [list, tuple, lambda v: np.array(v, dtype=object), np.array])
def test_ids_outside_the_vocabulary(bad, make):
    with pytest.raises(ValueError, match="outside the vocabulary of 100"):
        _token_ids(make([1, bad]), 100)


@pytest.mark.parametrize("tokens", [np.zeros((2, 2), dtype=np.int64), [[1, 2]], ["x"], [None]])
def test_what_is_no_row_of_ids(tokens):
    with pytest.raises((TypeError, ValueError)):
        _token_ids(tokens, 100)
