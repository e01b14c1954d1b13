"""Cells out of the reciprocals' range beside cells within it, bit for bit.

FP64: bricks of 8 cells per dimension that hold a field out of range send the warps whose
stencils reach them to the divides; a state with many such warps, and a split sweep, go to
kernels that divide everywhere.  Each RK4 step is compared with the oracle's step from the
same state, whose results are equal."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from sac_b200 import abi, problems

import _util

pytestmark = pytest.mark.gpu


def _steps_equal(P, nsteps, dt_frac=0.1, **sweep):
    """Steps the device; each of its steps against the oracle's from the device's state.
    Returns which steps ran the general form's own kernels."""
    c, o = _util.start(abi.Context, P), _util.start(Oracle, P)
    c.lib.sac_general_kernels.argtypes = [abi.ctypes.c_void_p]
    n, route = 2 * P.ndir + 2, []
    dt = dt_frac * o.getdt(0)
    c.getdt(0)
    for it in range(nsteps):
        for x in (c, o):
            x.advect(dt, it * dt, it, **sweep)
        got, want = c.download(), o.download()
        np.testing.assert_array_equal(_util.mesh(P, got)[..., :n], _util.mesh(P, want)[..., :n])
        route.append(c.lib.sac_general_kernels(c.h))
        o.upload(got)
    c.close()
    o.close()
    return route


def _problem(nx, ndir, sources, typ="periodic"):
    P = problems.random_problem(nx, ndir=ndir, seed=81, types=[typ] * (2 * len(nx)))
    if sources:
        P.params.eta, P.params.divbfix = 0.01, 1
    return P


def _tiny(P, cells, scale=1e-70):
    """Momentum and field of these cells (mesh indices) below 2^-200."""
    v = problems.var_index(P.ndir)
    for q in cells:
        c = tuple(slice(i + 2, i + 3) if np.ndim(i) == 0 else slice(i[0] + 2, i[1] + 2) for i in q)
        P.w[c][..., 1:1 + P.ndir] *= scale
        P.w[c][..., v["b0"] + 1:v["b0"] + 1 + P.ndir] *= scale


# single cells (mesh indices) at a brick's corner, on an edge and in an inner one, at the
# grid's first and last cell; bricks begin at the mesh indices 6, 14, 22, ...
CELLS = {2: [(14, 22), (29, 17), (0, 0), (42, 37)], 3: [(14, 22, 6), (29, 25, 17), (17, 14, 29), (0, 0, 0), (42, 37, 34)]}


@pytest.mark.parametrize("sources", [False, True])
@pytest.mark.parametrize("nx,ndir", [((43, 38), 2), ((43, 38, 35), 3)])
def test_split_sweeps_and_variable_lists(nx, ndir, sources):
    for kw in (dict(idimmin=2, idimmax=2), dict(iws=[1, 2, ndir + 2])):
        P = _problem(nx, ndir, sources)
        _tiny(P, CELLS[len(nx)])
        assert _steps_equal(P, 2, **kw) == [1, 1]
