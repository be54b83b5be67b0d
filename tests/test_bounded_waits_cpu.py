"""Bounded waits give up lane by lane.  A warp whose lanes then part - some leave a loop or the kernel, the others go on into a
warp-wide shuffle or barrier - never comes together again, and the bounded wait is a hang.  So no kernel may leave on one
lane's answer: a `break` or `return` that depends on a wait or on the abort flag takes a vote."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h100_gdn_cuda_b200", "csrc", "kernels")
LEAVES = re.compile(r"if \((?P<cond>.*(mbar_\w*wait\w*|abort_flag).*)\)\s*(\{\s*)?(break|return|continue)\b")
VOTE = re.compile(r"__(all|any)_sync\(|__syncthreads_or\(")


def lone_exits(text):
    text = re.sub(r"//[^\n]*", "", text)
    return [m.group(0) for m in map(LEAVES.search, text.splitlines()) if m and not VOTE.search(m.group("cond"))]


def test_the_rule_sees_a_lone_exit():
    assert lone_exits("if (!mbar_wait(&full[j], it & 1u, &abort_flag)) break;")
    assert lone_exits("if (*static_cast<volatile int*>(&abort_flag)) break;")
    assert not lone_exits("if (!__all_sync(0xffffffffu, mbar_wait(&full[j], it & 1u, &abort_flag))) break;")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(KERNELS) if f != "sm100_ptx.cuh"))
def test_no_lane_leaves_alone(name):
    with open(os.path.join(KERNELS, name)) as f:
        assert lone_exits(f.read()) == []
