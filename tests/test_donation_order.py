"""The order that the search's end rests on, read from its source (no GPU): the
lead lane counts the tasks that a warp is about to give away as outstanding, and
a warp barrier stands between that count and all that the donors do with them
(publish one, finish their own), so that the count of outstanding tasks cannot
reach 0 early."""
import os
import re

from conftest import PKG


def test_a_warp_barrier_follows_the_count_of_given_tasks():
    with open(os.path.join(PKG, "csrc", "search.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    count = src.index("atomicAdd(&ctl->outstanding, (uint32_t)__popc(donors))")
    publish = src.index("if (donor) {", count)
    between = src[count:publish]
    # outside the lead lane's branch, for the whole warp
    assert re.search(r"\}[^{}]*__syncwarp\(\);[^{}]*$", between), between
    assert "asm volatile" not in between  # an empty asm orders nothing on the device
