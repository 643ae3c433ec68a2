"""Segment counts that the wave model chooses for the fused products."""
from types import SimpleNamespace

import pytest

from igaops_b200.operators import FusedPlan


def _counts(tiles, groups, resident):
    return FusedPlan.predicted_nseg(SimpleNamespace(tiles=tiles, groups=groups, resident=resident))


@pytest.mark.parametrize("tiles", [1, 4, 9])
@pytest.mark.parametrize("groups", [1505, 6000, 21801])
def test_long_strips_are_cut_into_enough_segments(tiles, groups):
    """A strip of a few tiles: enough units to fill a third of the SMs' resident warps,
    or segments close to the shortest ones tried (eight groups)."""
    best = _counts(tiles, groups, 16)[0]
    assert tiles * best >= 148 * 16 / 3 or groups / best < 16


@pytest.mark.parametrize("groups", [1, 2, 3, 17, 130, 285, 513, 519, 520, 521, 527, 528, 100003])
def test_counts_are_distinct_and_leave_two_groups_a_segment(groups):
    counts = _counts(7, groups, 8)
    assert len(set(counts)) == len(counts) and min(counts) == 1
    assert max(counts) <= max(1, groups // 2)
    if groups <= 512:  # patches, not strips: every count up to 64
        assert sorted(counts) == list(range(1, max(1, min(64, groups // 2)) + 1))
