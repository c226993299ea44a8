"""The bound on the waits of the tensor-core kernels, as the header states it."""

import os
import re

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "atma_b200", "csrc", "sm100.cuh")


@pytest.mark.parametrize("gap", [1, 1000, 10 ** 6, 450_000_000, 900_000_000, 1_500_000_000, 2 ** 31 - 1])
def test_a_wait_that_runs_out_is_seen(gap):
    """Polls ``gap`` clocks apart, of a clock that starts over after 2^32: the difference passes the limit before twice the limit has gone by."""
    text = re.search(r"kWaitLimitClocks = ([^;]+);", open(HEADER).read()).group(1)
    limit = eval(text.replace("u", ""))                                     # an integer expression
    assert limit >= 10 ** 9                                                 # half a second at the highest clock: longer than any wait for work
    first = limit // gap + 1                                                # the first poll behind the limit
    assert first * gap < 2 ** 32 and (first * gap) % 2 ** 32 > limit
