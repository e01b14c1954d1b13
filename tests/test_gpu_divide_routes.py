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
from test_gpu_batch import _batch_of, _ot_problems

pytestmark = pytest.mark.gpu


def _steps_equal(P, nsteps, dt_frac=0.1, **sweep):
    """Steps the device; each of its steps against the oracle's from the device's state.
    Returns which steps ran the general form's own kernels."""
    c, o = _util.start(abi.Context, P), _util.start(Oracle, P)
    c.lib.sac_general_kernels.argtypes = [abi.ctypes.c_void_p]
    n, route = 2 * P.ndir + 2, []
    dt = dt_frac * o.getdt(0)
    for it in range(nsteps):
        c.getdt(it)  # brings the count that chooses the kernels
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
@pytest.mark.parametrize("nx,ndir", [((43, 38), 2), ((43, 38), 3), ((43, 38, 35), 3)])
def test_single_cells_out_of_range(nx, ndir, sources):
    """Six, six and five bricks per side: a cell's divides and its neighbours' fast form,
    each cell by itself and all together."""
    for cells in [[q] for q in CELLS[len(nx)]] + [CELLS[len(nx)]]:
        P = _problem(nx, ndir, sources)
        _tiny(P, cells)
        route = _steps_equal(P, 2)
        # away from the periodic ends a cell reaches 14 x 14 of the 38 x 35 rows
        if len(nx) == 3 and cells in [[q] for q in CELLS[3][:3]]:
            assert route == [0, 0]


@pytest.mark.parametrize("typ", ["periodic", "cont"])
@pytest.mark.parametrize("sources", ["none", "powell", "res", "all"])
@pytest.mark.parametrize("nx,ndir", [((43, 38), 2), ((43, 38), 3), ((43, 38, 35), 3)])
def test_many_cells_out_of_range(nx, ndir, sources, typ):
    """A state out of range in all but a corner: the first stage counts its warps and the
    steps after it run the general form's own kernels (not in 2D without sources)."""
    P = _problem(nx, ndir, False, typ)
    if sources in ("powell", "all"):
        P.params.divbfix = 1
    if sources in ("res", "all"):
        P.params.eta = 0.01
    v = problems.var_index(ndir)
    corner = tuple(slice(0, 9) for _ in nx)
    keep = P.w[corner].copy()
    P.w[..., 1:1 + ndir] *= 1e-70
    P.w[..., v["b0"] + 1:v["b0"] + 1 + ndir] *= 1e-70
    P.w[..., v["bg0"] + 1:] *= 1e-75
    P.params.grav[:] = [0.0, 0.0, 0.0]
    P.w[corner] = keep
    route = _steps_equal(P, 3)
    assert route[1:] == ([1, 1] if len(nx) == 3 or sources != "none" else [0, 0])


@pytest.mark.parametrize("sources", [False, True])
@pytest.mark.parametrize("nx,ndir", [((43, 38), 2), ((43, 38, 35), 3)])
def test_split_sweeps_and_variable_lists(nx, ndir, sources):
    for kw in (dict(idimmin=2, idimmax=2), dict(iws=[1, 2, ndir + 2])):
        P = _problem(nx, ndir, sources)
        _tiny(P, CELLS[len(nx)])
        assert _steps_equal(P, 2, **kw) == [1, 1]


@pytest.mark.parametrize("nx,cells", [(60, [(14,), (59,)]), (125, [(0,), (62,)]), (800, [(99,), (100,), (500,)]),
                                      (333, [((0, 333),)])])
def test_1d_step_with_cells_out_of_range(nx, cells):
    """The one-launch 1D step, cells at the ends of the clusters' segments among them."""
    P = _problem((nx,), 2, False)
    _tiny(P, cells)
    _steps_equal(P, 3)


@pytest.mark.parametrize("shape", [0, 1])
def test_fused_batch_stage_with_cells_out_of_range(shape):
    """A tile's one vote for its divides: the fused stage and the three passes, whose update
    divides everywhere, agree bit for bit."""
    Ps = _ot_problems([(40, 24), (64, 72), (70, 64)], [0.6, 2.5, 9.0])
    _tiny(Ps[0], [(31, 7)])
    _tiny(Ps[1], [(14, 22), (0, 0), (63, 71)])
    _tiny(Ps[2], [((0, 70), (0, 20))])
    a, f = (_batch_of(Ps, Ps[0].params) for _ in range(2))
    a.set_stage(False)
    f.set_stage(True, shape)
    for _ in range(3):
        a.advance(1)
        f.advance(1)
        np.testing.assert_array_equal(f.download(), a.download())


def test_a_state_that_leaves_rest_changes_kernels_in_a_step():
    """At rest every field is zero or background, which is in range, and the driver is zero
    in the step at t = 0; its far tail in the next is not. That step counts it and those
    behind it divide everywhere."""
    P = problems.stratified((48, 40, 40))
    P.params.userpar[4], P.params.userpar[6] = 0.03, 0.03  # out of range from 0.35 on
    assert _steps_equal(P, 4, dt_frac=0.5) == [0, 0, 1, 1]


@pytest.mark.parametrize("sources", [False, True])
@pytest.mark.parametrize("sheared", [False, True])
@pytest.mark.parametrize("nx,ndir", [((60,), 2), ((43, 38), 2), ((19, 18, 17), 3)])
def test_widths_out_of_range(nx, ndir, sheared, sources):
    """Widths beyond the reciprocals' range divide everywhere, with the table per axis and,
    where the axes are sheared, without any table."""
    P = _problem(nx, ndir, sources)
    P.params.grav[:] = [0.0, 0.0, 0.0]
    x = P.x * 1e15
    if sheared and len(nx) > 1:
        x[..., 0] *= 1.0 + 0.03 * P.x[..., 1]
    P.x = np.asfortranarray(x)
    if sources:
        P.params.eta *= 1e15
    route = _steps_equal(P, 2)
    if len(nx) > 1:
        assert route == [1, 1]
