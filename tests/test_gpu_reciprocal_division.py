"""The stage's divisions through reciprocals (qdiv) against the oracle's divides.

FP64: one RK4 step from the same state must equal the oracle's bit for bit on the
mesh (the background's drift enters only at the step's end), on grids whose widths
have a table per axis and on grids that need one per cell, and for states with cells
outside the range of the reciprocal form, which take the divide: subnormal, tiny
and huge fields beside ordinary ones."""
import numpy as np
import pytest

from sac_b200 import abi, params, problems

import _util

pytestmark = pytest.mark.gpu

SHAPES = [((40,), 2), ((21, 14), 2), ((21, 14), 3), ((11, 10, 9), 3)]


def _one_step(P, dt_frac=0.2, **sweep):
    from oracle.oracle import Oracle

    c, o = _util.start(abi.Context, P), _util.start(Oracle, P)
    dt = dt_frac * o.getdt(0)
    for x in (c, o):
        x.advect(dt, 0.0, 0, **sweep)
    got, want, n = c.download(), o.download(), 2 * P.ndir + 2
    c.close()
    o.close()
    return _util.mesh(P, got)[..., :n], _util.mesh(P, want)[..., :n]


def _problem(nx, ndir, sources):
    types = ["cont", "fixed", "periodic", "periodic", "cont1", "symm"][: 2 * len(nx)]
    P = problems.random_problem(nx, ndir=ndir, seed=51, types=types)
    if sources:
        P.params.eta, P.params.divbfix = 0.01, 1
    return P


def _stretch(P, tensor):
    """A smoothly stretched grid; not tensor: each axis also sheared along the others,
    so that no width depends on its own index alone."""
    x = P.x.copy(order="F")
    for d in range(P.ndim):
        s = x[..., d] + 0.05 * np.sin(2.0 * x[..., d])
        if not tensor:
            s = s * (1.0 + 0.03 * sum(P.x[..., e] for e in range(P.ndim) if e != d))
        x[..., d] = s
    P.x = np.asfortranarray(x)


@pytest.mark.parametrize("sources", [False, True])
@pytest.mark.parametrize("grid", ["uniform", "stretched", "sheared"])
@pytest.mark.parametrize("nx,ndir", SHAPES)
def test_step_equals_the_oracle_on_any_grid(nx, ndir, grid, sources):
    P = _problem(nx, ndir, sources)
    if grid != "uniform":
        _stretch(P, grid == "stretched")
    got, want = _one_step(P)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("scale", [5e-324, 3e-310, 1e-200, 1e-43, 1e31])
@pytest.mark.parametrize("nx,ndir", SHAPES)
def test_step_equals_the_oracle_with_cells_out_of_range(nx, ndir, scale):
    """The velocity and field of one half of the grid times `scale`, down to
    subnormals: tiles with such cells, tiles beside them and tiles without; and a
    state whose every value is huge."""
    P = _problem(nx, ndir, True)
    v = problems.var_index(ndir)
    half = (slice(None),) * (P.ndim - 1) + (slice(P.w.shape[P.ndim - 1] // 2, None),)
    w = P.w
    if scale > 1:  # the whole grid, the field by the root: the same wave speeds, and no
        w *= scale  # jump that would leave one side with a negative pressure
        w[..., v["b0"] + 1:v["b0"] + 1 + ndir] /= np.sqrt(scale)
        w[..., v["bg0"] + 1:] /= np.sqrt(scale)
    else:
        w[half][..., 0] = 0.0
        w[half][..., 1:1 + ndir] *= scale
        w[half][..., v["e"]] *= scale
        w[half][..., v["b0"] + 1:v["b0"] + 1 + ndir] *= scale
    got, want = _one_step(P, dt_frac=0.05)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("nx,ndir", SHAPES[1:])
def test_split_sweep_and_variable_list_equal_the_oracle(nx, ndir):
    """A dimensionally split sweep and a partial list of variables keep the general
    form of the update."""
    P = _problem(nx, ndir, True)
    for kw in (dict(idimmin=2, idimmax=2), dict(iws=[1, 2, ndir + 2])):
        got, want = _one_step(P, **kw)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("what", ["vacuum", "inf"])
@pytest.mark.parametrize("nx,ndir", SHAPES)
def test_fp32_infinities_are_the_quotients_own(nx, ndir, what):
    """FP32 storage: where a cell has no density or an infinite momentum, a stage's NaN
    and its infinities lie where the oracle's divides put them."""
    from oracle.oracle import Oracle

    P = problems.random_problem(nx, ndir=ndir, seed=52, nu=0.0, typeadvance="onestep")
    mid, rhob = tuple(n // 2 for n in P.w.shape[:-1]), problems.var_index(ndir)["rhob"]
    if what == "vacuum":
        P.w[mid][rhob], P.w[mid][0] = 1.0, -1.0
    else:
        P.w[mid][1] = np.inf
    o = _util.start(Oracle, P)
    P.params.precision = params.PREC_FP32
    c = _util.start(abi.Context, P)
    got, want = [], []
    for x, out in ((c, got), (o, want)):
        x.advect(1e-3, 0.0, 0)
        out.append(_util.mesh(P, x.download())[..., : 2 * ndir + 2])
        x.close()
    assert not np.isfinite(want[0]).all() and np.isfinite(want[0]).any()
    np.testing.assert_array_equal(np.isnan(got[0]), np.isnan(want[0]))
    np.testing.assert_array_equal(np.isinf(got[0]), np.isinf(want[0]))
