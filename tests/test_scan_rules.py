"""Which requests of a step go to the recurrences' kernel for portions of prompts."""

import pytest

from oxr_inference_b200 import ops

RULE = ops.ScanRule(least=16, beside=64, overlap=10)


@pytest.mark.parametrize("q_lens,want", [
    ([1] * 3, []), ([15, 15], []), ([16], [0]), ([700, 700], [0, 1]), ([16, 300, 17], [1, 2, 0]),          # all alike: by the length
    ([1] * 20 + [1200], [20]), ([1, 900, 15, 16, 1, 300], [1, 5, 3]),                                          # the portions alone, the longest first
    ([1] * 20 + [210], [20] + list(range(20))), ([1, 20], [1, 0]), ([1] * 20 + [211], [20]),                    # short against the number of others: all together
    ([1] * 40 + [63], []), ([1] * 40 + [64], [40]), ([1] * 40 + [17, 64, 15], [41, 40]), ([1, 21], [])])     # more than 32, or too short for a launch of their own
def test_which_requests(q_lens, want):
    """Single tokens beside a prompt do not count as its warps."""
    named, n = ops._long_requests(q_lens, sum(q_lens), len(q_lens), RULE)
    assert n == len(want) and list(named or ()) == want


def test_without_lengths_by_the_average():
    assert ops._long_requests(None, 128, 8, RULE) == (None, 8) and ops._long_requests(None, 127, 8, RULE) == (None, 0)


def test_lengths_of_another_step_are_refused():
    with pytest.raises(ops.KernelError, match="2 request lengths for 3 requests"):
        ops._long_requests([1, 5], 6, 3, RULE)
