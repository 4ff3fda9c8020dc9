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


def test_a_warp_waits_before_it_reads_the_instances_to_advance():
    """A lane leaves the instance it has finished an iteration of in shared
    memory, and all lanes of its warp read it: a vote is no barrier for memory,
    so a fence and a warp barrier come before each advance."""
    src = _source()
    vote = src.index("while (pend)", src.index("__ballot_sync(FULL, events & kAdvance)"))
    between = src[vote:src.index("warp_advance(P, s_cold0", vote)]
    assert re.search(r"\{\s*__threadfence\(\);\s*__syncwarp\(\);", between), between
