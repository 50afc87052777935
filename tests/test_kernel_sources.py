"""Properties of the kernel sources that no run shows: orderings between the lanes of a warp hold by luck until they do not."""
import os
import re

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


def test_every_lane_acquires():
    """A wait of a warp: a lane that learns of the phase from another (a shuffle, a vote) has acquired nothing and may read shared
    memory from before the copy it waited for, so every lane has to have tested the barrier itself."""
    b = body(open(os.path.join(CSRC, "lq_common.cuh")).read(), "warp_wait_bounded")
    assert "if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;" in b
    assert "lane" not in b and "shfl" not in b


def test_no_lane_waits_alone():
    """Nor does any other wait on a barrier hang on one lane."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
            if f == "lq_common.cuh":
                text = text.replace(body(text, "warp_wait_bounded"), "")
            for m in re.finditer(r"[^\n]*mbar_try_wait\([^\n]*", text):
                assert not re.search(r"if \((lane|tid|t|threadIdx\.x) ==", m.group(0)), (f, m.group(0).strip())
