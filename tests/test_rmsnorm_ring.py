"""Host side of the one-rank RMSNorm kernel: the ring of shared-memory slots that its groups of threads read rows from."""
import ctypes

import pytest


def _plan(lib, tokens, hidden, ctas):
    plan = (ctypes.c_int * 4)()
    assert lib.b200DevApiArRmsNormPlan(tokens, hidden, ctas, plan) == 0
    return plan[0], plan[1] // plan[0], plan[2], plan[3]


@pytest.mark.parametrize("ctas", [1, 3, 16, 64, 148, 1000])
def test_a_group_meets_every_use_of_its_slots(lib, ctas):
    """A wait on a slot's barrier tells two uses of the slot apart by one bit, so a group may wait for a use only when it has
    waited for the one before. Group g takes rows g, g + groups, ... of its CTA: it meets them all when a lap of the ring is a whole
    number of its steps, whatever order the copies land in. (No slot is used twice when a CTA's rows fit the ring.)"""
    for hidden in range(8, 16385, 8):
        for tokens in (0, 1, ctas, 5 * ctas + 3, 12 * ctas - 1, 12 * ctas, 17 * ctas, 32 * ctas + 1, 2048, 100003):
            group, groups, rows, stages = _plan(lib, tokens, hidden, ctas)
            at = (tokens, hidden, ctas, group, rows, stages)
            assert group * 8 >= hidden // 8, at                       # 8 packs of 8 channels per thread hold a row
            assert 1 <= stages <= 16 and rows >= 1 and 128 + stages * rows * hidden * 4 + hidden * 2 <= 227 * 1024 - 1024, at   # ring and gains
            assert stages * rows % groups == 0, at
