"""The one-launch RK4 step of small 1D grids against the oracle and against the launches.

Sizes around the cluster's segments (a last CTA with only ghost cells, one cell, an
empty one), the smallest and the first that do not take it, every default boundary
type and ndir, with and without hyperdiffusion, in both precisions.  FP64 equals the
oracle bit for bit after one step from the same state."""
import copy

import numpy as np
import pytest

from sac_b200 import abi, params, problems

import _util

pytestmark = pytest.mark.gpu


def _steps(P, cls, n, dts=None):
    c = _util.start(cls, P)
    dts = _util.run(c, n, dts=dts)
    w = _util.mesh(P, c.download())[..., : 2 * P.ndir + 2]
    k = c.lib.sac_kernel_launches(c.h) if cls is abi.Context else 0
    c.close()
    return w, dts, k


@pytest.mark.parametrize("nx,ndir,types", [
    (59, 1, ["cont", "symm"]), (60, 2, ["cont", "cont"]), (61, 2, ["periodic", "periodic"]),
    (68, 3, ["fixed", "asymm"]), (124, 2, ["symm0", "contCD4"]), (125, 2, ["cont1", "grad1"]),
    (800, 2, ["cont", "cont"]), (1021, 3, ["fixed1", "cont"]), (4000, 2, ["periodic", "periodic"])])
@pytest.mark.parametrize("visc", [True, False])
def test_step_equals_the_oracle(nx, ndir, types, visc):
    from oracle.oracle import Oracle

    P = problems.random_problem((nx,), ndir=ndir, seed=61, types=types)
    if not visc:
        P.params.nu = 0.0
    abi.load()[0].sac_kernel_launches.argtypes = [abi.ctypes.c_void_p]
    abi.load()[0].sac_kernel_launches.restype = abi.ctypes.c_long
    got, dts, k = _steps(P, abi.Context, 1)
    want, _, _ = _steps(P, Oracle, 1, dts)
    np.testing.assert_array_equal(got, want)
    # the 60-cell mesh is the smallest grid (64 cells) that takes the one launch
    if nx >= 60:
        assert k < 20, k
    got, dts, _ = _steps(P, abi.Context, 20)
    want, _, _ = _steps(P, Oracle, 20, dts)
    assert _util.rel_l2(got, want).max() <= 1e-12


def test_largest_grid_and_the_next_agree():
    """Two grids of one state, one just inside the cluster's shared memory and one that
    takes the launches: each against the oracle."""
    from oracle.oracle import Oracle

    for nx in (17000, 17600):
        P = problems.random_problem((nx,), ndir=2, seed=62, types=["periodic", "periodic"])
        got, dts, _ = _steps(P, abi.Context, 1)
        want, _, _ = _steps(P, Oracle, 1, dts)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("nx", [60, 333])
def test_fp32_steps_stay_in_the_twin_envelope(nx):
    P = problems.random_problem((nx,), ndir=2, seed=63, types=["cont", "cont"])
    err, twin = _util.fp32_twin(P, 4)
    assert (err <= 1e-5).all() or (err <= 150 * twin).all(), (err, twin)
    Q = copy.deepcopy(P)
    Q.params.precision = params.PREC_FP32
    w, _, _ = _steps(Q, abi.Context, 4)
    assert np.isfinite(w).all()


@pytest.mark.parametrize("fp32,most", [(False, 10000), (True, 17000)])
def test_the_largest_grid_of_one_launch_and_the_next(fp32, most):
    """The last grid (ghosts included) that takes the one launch and the first that takes
    the launches: FP64 equals the oracle, FP32 the other route's envelope."""
    from oracle.oracle import Oracle

    abi.load()[0].sac_kernel_launches.argtypes = [abi.ctypes.c_void_p]
    abi.load()[0].sac_kernel_launches.restype = abi.ctypes.c_long
    for n in (most, most + 1):
        P = problems.random_problem((n - 4,), ndir=3, seed=64, types=["periodic", "periodic"])
        if fp32:
            err, twin = _util.fp32_twin(P, 2)
            assert (err <= 1e-5).all() or (err <= 150 * twin).all(), (err, twin)
            P.params.precision = params.PREC_FP32
        got, dts, k = _steps(P, abi.Context, 1)
        assert (k < 10) == (n == most), (n, k)
        if not fp32:
            want, _, _ = _steps(P, Oracle, 1, dts)
            np.testing.assert_array_equal(got, want)
