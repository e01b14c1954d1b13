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


@pytest.mark.parametrize("name", ["fno_gemm.cuh", "fno_proj.cuh", "fno_row.cuh", "fno_wgrad.cuh"])
def test_a_bounded_wait_ends_alike_for_a_warp_before_it_loads_an_accumulator(name):
    """tcgen05.ld is executed by all lanes of a warp together, and a wait with a bound may
    end in time for some and not for others: a vote of the warp or of the block stands
    between every such load and the wait before it."""
    src = _code(os.path.join("fno", name))
    # (a wait whose result is not used lets products drain, with no load behind it)
    waits = [m.start() for m in re.finditer(r"(?<=!)mbar_wait\(|(?<=, )mbar_wait\(", src)]
    loads = [m.start() for m in re.finditer(r"tcgen05\.ld\.", src)]
    assert loads
    for ld in loads:
        wait = max(w for w in waits if w < ld)
        line = src.rindex("\n", 0, wait)
        assert re.search(r"__all_sync|__syncthreads_or", src[line:ld]), src[line:wait + 60]


def test_the_gemm_epilogue_gathers_its_warp_before_each_load():
    """The lanes of rows past M leave a turn of the column loop early; the next turn's load
    needs them back."""
    src = _code(os.path.join("fno", "fno_gemm.cuh"))
    turn = src[src.index("cc < BN"):]
    assert turn.index("__syncwarp()") < turn.index("tcgen05.ld") < turn.index("continue")


@pytest.mark.parametrize("name", ["sac_gpu.cu", "sac_batch.cu"])
def test_setting_a_grid_makes_no_pinned_allocation(name):
    """A pinned allocation and its release take over a millisecond each, several times the
    whole set-up of a small grid; what getdt brings to the host needs none."""
    assert not re.search(r"cudaMallocHost|cudaHostAlloc", _code(name))
