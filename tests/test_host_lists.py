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


def test_a_step_reads_short_lists_of_wanted_places_itself(monkeypatch):
    """A call of native code takes as long as some twenty numbers; both ways see the same places and refuse the same ones."""
    from nnis_b200.engine import SequenceStep
    from nnis_b200.engine.engine import Engine, StepError
    calls = []
    native = ops.list_to_ints
    monkeypatch.setattr(ops, "list_to_ints", lambda values, limit: calls.append(len(values)) or native(values, limit))

    class Cache:
        groups = ()
        length = staticmethod(lambda slot: 0)
        reserve = staticmethod(lambda slots, lengths: None)

    class Anything:
        vocab_size = 64
        device = torch.device("cpu")
        step_tables = staticmethod(lambda counts, starts: {})
    engine = Engine.__new__(Engine)
    engine.spec = engine.model = Anything
    engine.cache, engine.device = Cache, Anything.device
    engine._stage = lambda parts, workspace: torch.from_numpy(np.concatenate([p.reshape(-1) for p in parts]))
    prepare = lambda tokens, want: engine.prepare([SequenceStep(0, [1, 2, 3], [2]), SequenceStep(1, tokens, want)], object())[1].tolist()
    tokens = list(range(40))
    for want in ([], [0, 39], list(range(23)), list(range(0, 40)), tuple(range(40)), np.arange(5), [True, np.int64(7)]):
        calls.clear()
        assert prepare(tokens, want) == [2] + [3 + int(w) for w in want]
        assert calls == [3, 40] + ([40] if type(want) is list and len(want) >= 24 else [])
    for want in ([40], [-1], [0] * 30 + [40], [0] * 30 + [-1]):
        with pytest.raises(StepError, match="wanted place"):
            prepare(tokens, want)
    for bad in ([64], [-1], [0] * 30 + [64]):
        with pytest.raises(StepError, match="outside the vocabulary"):
            prepare(bad, [0])
    with pytest.raises(StepError, match="at least one token"):
        prepare([], [])
