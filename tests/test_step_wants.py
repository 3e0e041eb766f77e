"""The places a step's entries want: anything that has a length and can be gone through, checked before the step begins."""
import numpy as np
import pytest

from cajeta_llm_b200.engine.step import StepEntry, StepError, wanted_places


@pytest.mark.parametrize("want", [[1, 4], (1, 4), range(1, 5, 3), {1, 4}, {1: "a", 4: "b"}, {1: "a", 4: "b"}.keys(), np.array([1, 4]), np.array([1, 4], np.uint8),
                                  [np.int32(1), 4]])
def test_any_collection_of_places(want):
    entries = [StepEntry(0, [7] * 5, want), StepEntry(1, [7], ()), StepEntry(2, [7] * 2, [1])]
    n, places = wanted_places(entries, np.array([5, 1, 2], np.int32))
    assert n.tolist() == [2, 0, 1] and places.dtype == np.int32
    assert sorted(places[:2].tolist()) == [1, 4] and places[2] == 1


def test_no_places():
    n, places = wanted_places([StepEntry(0, [7]), StepEntry(1, [7, 8], [])], np.array([1, 2], np.int32))
    assert n.tolist() == [0, 0] and places.shape == (0,)


@pytest.mark.parametrize("want", [[5], {-1}, [0, 2 ** 31 + 1], [2 ** 70], [-2 ** 70]])
def test_places_outside_the_tokens_are_refused(want):
    with pytest.raises(StepError):
        wanted_places([StepEntry(0, [7] * 9, [8]), StepEntry(1, [7] * 5, want)], np.array([9, 5], np.int32))
