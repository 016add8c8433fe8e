"""A step's tokens as an array: what is taken in one go, what is left to the general path, and that neither refuses or lets
through what the other does not; wanted places spread over the chunks of a long step."""
import numpy as np
import pytest

from cpp_minilamma_b200.engine.step import Engine, StepEntry, StepError, _whole_numbers


class _Cache:
    seq_len = [5]

    def is_live(self, slot):
        return slot == 0

    def reserve(self, growth):
        self.growth = growth


def _planner(limit):
    engine = Engine.__new__(Engine)  # planning alone: no model, no device
    engine.vocab_size, engine.max_step_tokens, engine.cache = 100, limit, _Cache()
    return engine


@pytest.mark.parametrize("tokens,taken", [
    ([1, 2, 3], True), ([np.int32(4), True], True), (np.arange(3, dtype=np.int32), True), (np.arange(3), True),
    ((1, 2), False), ([1.5, 2], False), ([1 << 70], False), (np.zeros((2, 2), dtype=np.int64), False),
    (np.array([0.0, 1.0]), False), (range(3), False)])
def test_whole_numbers(tokens, taken):
    values = _whole_numbers(tokens)
    assert (values is not None) == taken
    if taken:
        assert values.tolist() == [int(t) for t in tokens]


@pytest.mark.parametrize("bad", [[3, -1], [100], [1 << 70], np.array([7, 100]), (5, -2), [-0.5]])
def test_refused_tokens(bad):
    with pytest.raises(StepError, match="outside the vocabulary"):
        _planner(64)._plan([StepEntry(0, bad)])


@pytest.mark.parametrize("kind", [list, tuple, np.array])
def test_chunks_and_wanted_places(kind):
    tokens = list(range(50))
    chunks, n_want = _planner(20)._plan([StepEntry(0, kind(tokens), [49, 0, 19, 20, 0])])
    assert n_want == 5
    assert [t for chunk in chunks for seq in chunk for t in seq.tokens] == tokens
    assert [seq.start for chunk in chunks for seq in chunk] == [5, 25, 45]
    assert [seq.want for chunk in chunks for seq in chunk] == [[(0, 1), (0, 4), (19, 2)], [(0, 3)], [(9, 0)]]


def test_wanted_places_are_walked_once():
    """A prompt in many chunks with every place wanted: the planning compares each place with a few others, not with every chunk."""
    compared = [0]

    class Place(int):
        def __lt__(self, other):
            compared[0] += 1
            return int(self) < int(other)

        def __le__(self, other):
            compared[0] += 1
            return int(self) <= int(other)

        def __gt__(self, other):
            compared[0] += 1
            return int(self) > int(other)

        def __ge__(self, other):
            compared[0] += 1
            return int(self) >= int(other)

        __eq__, __hash__ = int.__eq__, int.__hash__

    n = 2000
    chunks, n_want = _planner(20)._plan([StepEntry(0, [1] * n, [Place(i) for i in range(n)])])
    assert n_want == n and len(chunks) == n // 20
    assert [seq.want for chunk in chunks for seq in chunk] == [[(i, c * 20 + i) for i in range(20)] for c in range(n // 20)]
    assert compared[0] < 20 * n
