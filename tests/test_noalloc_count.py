"""The counter that a search without allocation leaves: what a caller makes of
it. The header names the bit of a wait that ran out, and the kernel sets that."""
import os
import re

import pytest

from onion_gen_b200 import _native as N
from onion_gen_b200 import gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_bit_is_in_the_header():
    text = open(os.path.join(ROOT, "include", "onion_gen_b200.h")).read()
    assert int(re.search(r"#define OG_NOALLOC_FAILED (0x[0-9a-f]+)u", text).group(1), 16) == N.NOALLOC_FAILED


@pytest.mark.parametrize("count", [0, 1, 100])
def test_records(count):
    assert gpu.noalloc_records(count, 100) == count


@pytest.mark.parametrize("count,status", [(101, "OG_E_OVERFLOW"), (2**31 - 1, "OG_E_OVERFLOW"),
                                          (N.NOALLOC_FAILED, "OG_E_TIMEOUT"), (N.NOALLOC_FAILED + 5, "OG_E_TIMEOUT"),
                                          (-(2**31), "OG_E_TIMEOUT"), (5 - 2**31, "OG_E_TIMEOUT")])
def test_what_is_no_result(count, status):
    """A signed word with the bit set is negative: not an empty result."""
    with pytest.raises(N.OgError) as e:
        gpu.noalloc_records(count, 100)
    assert e.value.status == status
