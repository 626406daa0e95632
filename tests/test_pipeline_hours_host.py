"""Ranges of hours of the batched day's sweep stage."""
import inspect

import pytest


@pytest.mark.parametrize("given,want", [
    (0, None), (5, [(0, 5), (5, 10), (10, 15), (15, 20), (20, 24)]), ((20, 3), [(0, 20), (20, 23), (23, 24)]),
    ((2, 2, 2, 2, 4, 4, 8), [(0, 2), (2, 4), (4, 6), (6, 8), (8, 12), (12, 16), (16, 24)])])
def test_ranges_depend_on_the_values_given(given, want):
    from solweig_cuda_b200 import batched
    assert batched.ChosenDay._ranges(24, given) == want
    if want is not None and not isinstance(given, int):
        assert batched.ChosenDay._ranges(24, list(given)) == want


def test_a_day_is_one_range_by_default():
    from solweig_cuda_b200 import batched
    default = inspect.signature(batched.ChosenDay.__init__).parameters["pipeline_hours"].default
    assert batched.ChosenDay._ranges(24, default) is None
