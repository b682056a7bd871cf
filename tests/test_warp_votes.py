"""Roles of the tensor-core kernels whose warps vote: a lane must not leave its warp after a wait of its own.

A bounded wait may end differently in the lanes of a warp (each polls and reads the clock for itself). Where a role then votes over the whole warp, or waits
as a whole warp, only if it is still alive, the lanes that gave up never arrive at the vote and the others stay in it without a limit. So such a role takes its
answers from the waits that vote themselves. Nothing here needs a device: the roles are read from the source.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xn_b200", "csrc")


def _roles(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    return re.split(r"\bbool alive = true", text)[1:]


@pytest.mark.parametrize("name,roles", [("xnq_prefill.cu", 5), ("xnq_imma.cu", 5)])
def test_a_role_that_votes_waits_as_a_warp(name, roles):
    blocks = _roles(name)
    assert len(blocks) == roles
    for block in blocks:
        lane_by_lane = re.search(r"\balive = mbar_wait\(", block)
        conditional_vote = re.search(r"\balive &&[^;{]*__all_sync|\balive = mbar_wait_(warp|uniform)\(", block)
        assert not (lane_by_lane and conditional_vote), f"{name}: {lane_by_lane.group(0)} in a role with {conditional_vote.group(0)}"
