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


@pytest.mark.parametrize("width,B", [(32, 32), (64, 64)])
def test_a_smaller_network_beside_a_larger_one(width, B):
    """The mode mixing's shared memory follows max_batch: a network of one sample made
    later leaves the larger one its launches."""
    torch = pytest.importorskip("torch")
    from sac_b200 import fno_abi

    S = F = 56
    net = fno_abi.Net(S=S, F=F, width=width, layers=1, max_batch=B, seed=5)
    x = torch.randn(B, 16, S, F, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    dy = torch.zeros(B, net.cpad, S, F, dtype=torch.bfloat16, device="cuda")
    dy[:, :6] = 1e-3
    y = [torch.zeros(B, 6, S, F, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    grads = []
    for k in range(2):
        net.zero_grad()
        net.forward(x.data_ptr(), y[k].data_ptr(), B)
        if width == 32:  # the wider network trains on smaller batches only
            net.backward(dy.data_ptr())
        net.check()
        grads.append(net.get_grads())
        other = fno_abi.Net(S=S, F=F, width=width, layers=1, max_batch=1, seed=6)
    assert torch.equal(y[0], y[1])
    # sums of atomic additions, in another order from run to run
    assert np.linalg.norm(grads[0] - grads[1]) <= 1e-4 * np.linalg.norm(grads[0]) + 1e-30
    other.close()
    net.close()
