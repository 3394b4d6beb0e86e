"""The autotuner times every bucket of the table at a count that lies in it."""
import math

import pytest

import mdiscriminator_b200 as mdx
from mdiscriminator_b200 import autotune


@pytest.mark.parametrize("elem", [mdx.ELEM_U32, mdx.ELEM_REC8])
def test_timed_counts_lie_in_their_buckets(elem):
    for n, (lo, hi) in autotune.BUCKETS:
        assert lo <= math.ceil(math.log2(autotune.timed_count(elem, n, (lo, hi)))) <= hi
    bounds = [b for _, b in autotune.BUCKETS]
    assert bounds[0][0] == 0 and bounds[-1][1] == 33
    assert all(a[1] + 1 == b[0] for a, b in zip(bounds, bounds[1:]))
