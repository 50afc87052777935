"""Properties of the kernel sources that no run shows: orderings between the lanes of a warp hold by luck until they do not."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "leapquant_b200", "csrc")


def body(text, name):
    """The braces of the function `name`, without comments."""
    text = re.sub(r"//[^\n]*", "", text)
    at = text.index("{", text.index(f" {name}("))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]


@pytest.mark.parametrize("name", ["warp_wait_bounded"])
def test_broadcast_wait_orders_the_warp(name):
    """One lane tests the barrier and a shuffle tells the others, which orders no memory: before the function reports success the
    warp has to synchronise, or the other lanes may read shared memory from before the copy they waited for."""
    b = body(open(os.path.join(CSRC, "lq_common.cuh")).read(), name)
    poll, told, sync, done = (b.index(s) for s in ("mbar_try_wait(", "__shfl_sync(", "__syncwarp()", "return true"))
    assert poll < told < sync < done


def test_one_lane_waits_only_through_it():
    """Every other wait on a barrier is one that each thread makes for itself."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
            if f == "lq_common.cuh":
                text = text.replace(body(text, "warp_wait_bounded"), "")
            for m in re.finditer(r"[^\n]*mbar_try_wait\([^\n]*", text):
                assert not re.search(r"if \((lane|tid|t|threadIdx\.x) ==", m.group(0)), (f, m.group(0).strip())
