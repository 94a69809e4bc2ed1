"""The warp walk's stacks (dr_walk_rules.cuh) on the CPU: their pushes are not
checked, so the rules that class the pending nodes and pick a step's nodes have
to keep every stack within its entries, also when no node can be handed on
(the packet queue is full) and whatever the nodes' shares are, undefined ones
(NaN) among them."""
import numpy as np
import pytest

from native import harness

SIZES = np.array([128, 128, 224])  # DR_WALK_N0, N1, N2


@pytest.mark.parametrize("levels", [6, 28])
@pytest.mark.parametrize("child", [60, 75, 97])
@pytest.mark.parametrize("split", [0, 50, 90])
def test_stacks_hold_walks_that_cannot_be_handed_on(levels, child, split):
    most = np.zeros(3, np.int64)
    crowded = 0
    for off in (0, 5, 60):
        for nan in (0, 10, 90):
            held, steps = harness.walk_stacks(levels + child + split + off + nan, 4, levels, child, split, off, nan)
            most = np.maximum(most, held)
            crowded += steps
    assert (most <= SIZES).all(), most
    if levels == 28 and child > 60:
        assert crowded > 1000  # the branch without room is taken
        assert most[0] > 96 and most[1] > 96  # and the reserve is used
