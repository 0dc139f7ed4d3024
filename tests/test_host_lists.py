"""Token lists read by native code: the same numbers as numpy's, and None for whatever a caller has to look at itself."""
import numpy as np
import pytest
import torch

from nnis_b200.csrc import ops


@pytest.mark.parametrize("n", [0, 1, 2, 1000])
def test_lists_of_whole_numbers(n):
    values = [int(v) for v in np.random.default_rng(n).integers(0, 49152, n)]
    got = ops.list_to_ints(values, 49152)
    assert got.dtype == np.int32 and got.tolist() == values
    assert ops.list_to_ints([True, np.int64(7), torch.tensor(3)], 8).tolist() == [1, 7, 3]


@pytest.mark.parametrize("values", [[-1], [0, 8], [1, 2.0], [None], ["1"], [2 ** 40], [-2 ** 70], [2 ** 70], [[1]], [np.float32(1)]])
def test_what_is_left_to_the_caller(values):
    assert ops.list_to_ints(values, 8) is None
    assert ops.list_to_ints([1, 2], 8).tolist() == [1, 2]  # (no error is left behind)


def test_a_number_that_changes_the_list_or_fails():
    class Shrinks:
        def __init__(self, values):
            self.values = values

        def __index__(self):
            del self.values[1:]
            return 1

    class Fails:
        def __index__(self):
            raise RuntimeError("no")

    values = []
    values += [Shrinks(values), 1, 2]
    assert ops.list_to_ints(values, 8) is None
    assert ops.list_to_ints([Fails()], 8) is None and ops.list_to_ints([3], 8).tolist() == [3]
