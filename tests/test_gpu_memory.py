"""The device memory of a single grid, counted from its fields."""
import pytest

from sac_b200 import abi, params, problems

import _util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _sheared(P):
    x = P.x.copy(order="F")
    x[..., 0] *= 1.0 + 0.03 * P.x[..., 1]
    P.x = x


@pytest.mark.parametrize("sheared", [False, True])
@pytest.mark.parametrize("nx,ndir", [((1024, 768), 2), ((96, 96, 96), 3)])
def test_fp32_grid_holds_its_fields_and_no_more(nx, ndir, sheared):
    """Four states of np fields, nw - np background fields (64 bits), the stage's D, F and
    R, the widths (64 bits), one of coordinates (64 bits) that a table of widths per cell
    may take instead, and the staging block of the upload (64 bits); the cross terms share
    that block."""
    P = problems.random_problem(nx, ndir=ndir, seed=5)
    if sheared:
        _sheared(P)
    P.params.precision = params.PREC_FP32
    nd, np_ = len(nx), 2 * ndir + 2
    cells = 1
    for n in nx:
        cells *= n + 4
    pairs = 2 * nd + nd * nd + nd * (nd - 1)
    per_cell = 4 * (4 * np_ + (ndir + 3) + nd * np_ + pairs) + 8 * ((ndir + 2) + 2 * nd + np_)
    _util.start(abi.Context, P).close()  # the library and its kernels are loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    c = _util.start(abi.Context, P)
    used = free - torch.cuda.mem_get_info()[0]
    c.close()
    # fixB and the small tables, and the allocations' rounding to 2 MB
    assert used <= per_cell * cells * 1.02 + 40e6, (used, per_cell * cells)


def test_a_network_of_the_row_kernel_holds_no_fp32_intermediates():
    """Activations, pre-activations, dz and its twin (BF16), the three hidden buffers (BF16),
    the transforms and the parameters: no FP32 buffer of width x pixels."""
    from sac_b200 import fno_abi

    B, S, F, W, L, H, kJ, kR = 8, 256, 256, 32, 4, 128, 48, 96
    bwp = B * W * S * F
    fno_abi.Net(S=S, F=F, max_batch=1, seed=1).close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    net = fno_abi.Net(S=S, F=F, max_batch=B, seed=1)
    used = free - torch.cuda.mem_get_info()[0]
    npar = net.nparam
    net.close()
    want = 2 * bwp * ((L + 1) + L + 2 + 3 * H // W) + 4 * 2 * B * W * kJ * S + (4 * (L + 1) + 2 * 2) * B * W * kJ * kR
    assert used <= (want + 18 * npar) * 1.02 + 40e6, (used, want + 18 * npar)
