"""Objects of different sizes side by side: each must give what it gives alone.

The kernels' launch attributes belong to the process, so a size that one object sets must
not be what another one launches with."""
import threading

import numpy as np
import pytest

from sac_b200 import abi, problems

import _util

pytestmark = pytest.mark.gpu


def test_1d_grids_of_different_sizes_in_their_threads():
    """One context per host thread: a grid whose cluster takes over 100 KB of shared memory
    per CTA beside three that take a few, stepped at the same time."""
    large, small, nsteps = 8000, 60, 3000
    problem = {n: problems.random_problem((n,), ndir=2, seed=71, types=["periodic", "periodic"]) for n in (large, small)}
    out, err, done = {}, [], threading.Event()

    def steps(n, until=None):
        c = _util.start(abi.Context, problem[n])
        for it in range(nsteps):
            c.advect(1e-7, 0.0, it)
        w = c.download()
        while until and not until.is_set():  # keep launching while the large grid runs
            c.advect(1e-7, 0.0, nsteps)
        c.close()
        return w

    def thread(key, n, until=None):
        try:
            out[key] = steps(n, until)
        except Exception as e:
            err.append((n, e))
        finally:
            if until is None:
                done.set()

    alone = {n: steps(n) for n in problem}
    ts = [threading.Thread(target=thread, args=(k, small, done)) for k in range(3)]
    ts.append(threading.Thread(target=thread, args=(3, large)))
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not err, err
    for k in range(4):
        np.testing.assert_array_equal(out[k], alone[large if k == 3 else small])
