"""The segment planner as the operator asks it for K = V = 128: segments from four chunks on, and a fixed
cost of splitting at all.  Against the restated rule of test_planner.py."""

import random

import pytest
from test_planner import _plan


@pytest.mark.parametrize("seed", range(8))
def test_short_segments_and_a_fixed_cost(seed):
    from flashqla_b200 import _lib

    rng = random.Random(seed)
    heads = rng.choice([1, 2, 4, 8, 32])
    bounds = [0]
    for _ in range(rng.choice([1, 2, 7, 30])):
        bounds.append(bounds[-1] + rng.choice([0, 1, 63, 64, 65, 511, 512, rng.randint(1, 6000)]))
    split = _lib.host().split_sequences
    assert split(bounds, heads, 148, 4, 1) == split(bounds, heads, 148, 4, 1, 0) == _plan(bounds, heads, 148, 4)
    # the fixed cost changes whether a batch is split, never how
    assert split(bounds, heads, 148, 4, 1, 4) in (None, _plan(bounds, heads, 148, 4))
    assert split(bounds, heads, 148, 4, 1, 10**6) is None


def test_the_operators_constants():
    """One prompt on 8 heads: 64 chunks go to segments of four, eight chunks are left alone."""
    from flashqla_b200 import _lib

    split = _lib.host().split_sequences
    assert split([0, 64 * 64], 8, 148, 4, 1, 4) == ([64 * 4 * i for i in range(17)], [0, 16])
    assert split([0, 64 * 8], 8, 148, 4, 1, 4) is None
    assert split([0, 64 * 7], 8, 148, 4, 1, 0) is None
