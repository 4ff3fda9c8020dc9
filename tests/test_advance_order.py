"""The order that an instance's advance rests on, read from its source (no GPU)."""
import os
import re

from conftest import PKG


def _source():
    with open(os.path.join(PKG, "csrc", "search.cu")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_a_warp_barrier_follows_the_count_of_an_iterations_tasks():
    """Lane 0 counts the next iteration's tasks as outstanding, all lanes publish
    them: the barrier stands between the two, for the whole warp, so that no
    task can be finished before it was counted."""
    src = _source()
    count = src.index("atomicAdd(&ctl->outstanding, na + na2)")
    between = src[count:src.index("publish_root(P, t0 + b", count)]
    assert re.search(r"__shfl_sync\([^;]*;\s*__syncwarp\(\);\s*for \(", between), between
