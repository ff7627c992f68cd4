"""A barrier wait that can run out is made by one thread, or by a whole warp that gives up as one (mbar_wait_warp): after a wait that
ran out in some lanes alone, the others would stay at the next shuffle or warp barrier for good. That cannot be provoked
without hanging a GPU, so the sources are held to it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "outbreaklab_b200", "csrc")

# the barriers that single threads wait for (TMA producers, MMA issuers), and those that whole warps wait for
WAITS = {
    "ob_dst_tc.cu": ({"&empty[s]", "&tempty[b]", "&full[s]", "done", "bar"}, {"&tfull[b]"}),
    "ob_mlp_train_tc.cu": ({"wbar", "&empty[s]", "&full[s]", "ok ? bar : wbar"}, {"bar", "accf"}),
}


@pytest.mark.parametrize("name", sorted(WAITS))
def test_waits_of_warps_end_as_one(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    one = set(re.findall(r"\bmbar_wait\(([^,]+),", src))
    warp = set(re.findall(r"\bmbar_wait_warp\(([^,]+),", src))
    assert (one, warp) == WAITS[name]
    for m in re.finditer(r"\bmbar_wait\(", src):   # each in a branch that one thread takes
        before = src[:m.start()]
        depth, guarded = 0, False
        for k in range(len(before) - 1, 0, -1):
            if before[k] == "}":
                depth += 1
            elif before[k] == "{":
                if depth:
                    depth -= 1
                elif re.search(r"(lane == 0|tid == 0)[^;{}]*\{$", before[:k + 1]):
                    guarded = True
                    break
            if before[k] == "\n" and depth == 0 and re.search(r"(lane == 0|tid == 0)\)[^\n]*$", before[k:]):
                guarded = True
                break
            if before[k:].startswith("__global__"):
                break
        assert guarded, before[-200:]
