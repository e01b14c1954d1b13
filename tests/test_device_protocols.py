"""Orders in the device code that no run can be relied on to show, read from the source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sac_b200", "csrc")


def _code(name):
    """The source of one file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


@pytest.mark.parametrize("name", ["sac_step1d.cuh"])
def test_distributed_shared_memory_is_reached_after_a_cluster_barrier(name):
    """A CTA may touch another's shared memory only once every CTA of the cluster has
    started, which a barrier of the cluster shows: its wait comes before the first access,
    and each arrival has its wait."""
    src = _code(name)
    access = src.index("map_shared_rank")
    wait = re.search(r"cluster\.(sync|barrier_wait)\(\)", src)
    assert wait and wait.start() < access
    assert src.count("barrier_arrive()") == src.count("barrier_wait()")
