"""The FNO's row kernel and its vectorised streaming kernels at the edges of their ranges.

Forward passes against the float64 oracle on grids with one and two pixel tiles per
row, ragged rows, few and many rows per CTA, and just past the row kernel's width (one
GEMM per product); the bound is the one of the BF16 network (2e-2 relative L2)."""
import numpy as np
import pytest

from oracle import fno_ref

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _net(S, F, B):
    from sac_b200 import fno_abi

    return fno_abi.Net(S=S, F=F, max_batch=B, seed=3)


@pytest.mark.parametrize("S,F,B", [(56, 56, 1), (56, 128, 1), (64, 136, 3), (200, 120, 5), (104, 248, 2), (64, 256, 1),
                                   (56, 264, 1)])
def test_forward_matches_the_oracle(S, F, B):
    net, lay = _net(S, F, B), fno_ref.Layout(32, 4, 16, 6, 128)
    x = torch.randn(B, 16, S, F, generator=torch.Generator().manual_seed(9)).to(torch.bfloat16)
    xd, y = x.cuda(), torch.full((B, 6, S, F), float("nan"), device="cuda")
    y2 = y.clone()
    torch.cuda.synchronize()
    net.forward(xd.data_ptr(), y.data_ptr(), B)
    net.infer(xd.data_ptr(), y2.data_ptr(), B)
    net.check()
    theta = net.get_params().astype(np.float64)
    # the network reads BF16 weights (biases stay FP32)
    for name, (o, n) in lay.segs.items():
        if not name.endswith("b") and not (name[-1].isdigit() and name.startswith("Wb")):
            theta[o:o + n] = fno_ref.bf16_round(theta[o:o + n])
    want, _ = fno_ref.forward(lay, theta, x.double().numpy())
    got = y.cpu().double().numpy()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 2e-2
    assert torch.equal(y, y2)


def test_unaligned_buffers_give_the_same():
    """features and apply with buffers off the 16-byte boundary take the scalar
    kernels: the same values (the loss up to the order of its sum)."""
    S, F, B = 56, 72, 2
    net = _net(S, F, B)
    g = torch.Generator("cuda").manual_seed(4)

    def buf(shape, dtype, off):
        n = int(np.prod(shape))
        return torch.zeros(n + off, dtype=dtype, device="cuda")[off:].view(shape)

    st = torch.randn(B, 6, S, F, generator=g, device="cuda")
    sc, feat = torch.rand(B * 6, generator=g, device="cuda"), torch.rand(B * 4, generator=g, device="cuda")
    y, t = torch.randn(B, 6, S, F, generator=g, device="cuda"), torch.randn(B, 6, S, F, generator=g, device="cuda")
    out = []
    for off in (0, 1):
        s, yy = buf(st.shape, torch.float32, off), buf(y.shape, torch.float32, off)
        tt = buf(t.shape, torch.bfloat16, off)
        x, dy = buf((B, 16, S, F), torch.bfloat16, off), buf((B, 8, S, F), torch.bfloat16, off)
        s.copy_(st), yy.copy_(y), tt.copy_(t)
        loss = torch.zeros(1, device="cuda")
        torch.cuda.synchronize()
        net.features(s.data_ptr(), False, sc.data_ptr(), feat.data_ptr(), 4, x.data_ptr(), B, 6)
        net.apply(s.data_ptr(), yy.data_ptr(), sc.data_ptr(), B, 6)
        net.mse(yy.data_ptr(), tt.data_ptr(), dy.data_ptr(), loss.data_ptr(), B)
        net.check()
        torch.cuda.synchronize()
        out.append((x.clone(), s.clone(), dy.clone(), float(loss)))
    for a, b in zip(out[0][:3], out[1][:3]):
        assert torch.equal(a, b)
    # FP32 sums of 48384 squares in another order: n^0.5 * 2^-24 relative, with room
    assert abs(out[0][3] - out[1][3]) <= 1e-4 * abs(out[1][3])


@pytest.mark.parametrize("S,F,B", [(56, 56, 1), (56, 128, 1), (64, 136, 3), (200, 120, 5), (104, 248, 2), (64, 256, 1),
                                   (56, 264, 1)])
def test_gradients_match_the_oracle(S, F, B):
    """Every gradient group within the BF16 network's bound (5e-2 relative L2)."""
    net, lay = _net(S, F, B), fno_ref.Layout(32, 4, 16, 6, 128)
    g = torch.Generator().manual_seed(10)
    x = torch.randn(B, 16, S, F, generator=g).to(torch.bfloat16)
    dy = torch.zeros(B, net.cpad, S, F)
    dy[:, :6] = torch.randn(B, 6, S, F, generator=g)
    dy = dy.to(torch.bfloat16)
    xd, dyd, y = x.cuda(), dy.cuda(), torch.zeros(B, 6, S, F, device="cuda")
    torch.cuda.synchronize()
    net.zero_grad()
    net.forward(xd.data_ptr(), y.data_ptr(), B)
    net.backward(dyd.data_ptr())
    net.check()
    got = net.get_grads().astype(np.float64)
    theta = net.get_params().astype(np.float64)
    for name, (o, n) in lay.segs.items():
        if not name.endswith("b") and not (name[-1].isdigit() and name.startswith("Wb")):
            theta[o:o + n] = fno_ref.bf16_round(theta[o:o + n])
    _, tape = fno_ref.forward(lay, theta, x.double().numpy())
    want = fno_ref.backward(lay, theta, tape, dy[:, :6].double().numpy())
    for name, (o, n) in lay.segs.items():
        if name in ("Q2", "Q2b"):
            n = 6 * (128 if name == "Q2" else 1)
        err = np.linalg.norm(got[o:o + n] - want[o:o + n]) / np.linalg.norm(want[o:o + n])
        assert err < 5e-2, (name, err)


@pytest.mark.parametrize("B", [1, 64])
def test_the_transform_wait_running_out_is_reported(B):
    """The wait for the product with G, which a CTA reaches after each task of four rows
    (one task per CTA, and several): sac_fno_check returns 7, and the network gives what it
    gave before once the default bound is back."""
    from sac_b200 import fno_abi

    S, F = 56, 72
    net = _net(S, F, B)
    x = torch.randn(B, 16, S, F, generator=torch.Generator().manual_seed(9)).to(torch.bfloat16).cuda()
    y = [torch.zeros(B, 6, S, F, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    net.infer(x.data_ptr(), y[0].data_ptr(), B)
    net.check()
    net.set_t_wait_tries(-1)
    net.infer(x.data_ptr(), y[1].data_ptr(), B)
    with pytest.raises(fno_abi.FnoError) as e:
        net.check(reset=True)
    assert "status 7" in str(e.value)
    net.set_t_wait_tries(0)
    net.infer(x.data_ptr(), y[1].data_ptr(), B)
    net.check(reset=True)
    assert torch.equal(y[0], y[1])
    net.close()


def test_no_samples_and_no_state_channels_are_no_work():
    """features and apply of no samples, and apply of no channels, leave everything as it is."""
    S, F = 56, 72
    net = _net(S, F, 1)
    st, sc = torch.ones(6, S, F, device="cuda"), torch.ones(6, device="cuda")
    x = torch.ones(16, S, F, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    for bf16 in (False, True):
        net.features(st.data_ptr(), bf16, sc.data_ptr(), sc.data_ptr(), 4, x.data_ptr(), 0, 6)
    net.apply(st.data_ptr(), st.data_ptr(), sc.data_ptr(), 0, 6)
    net.apply(st.data_ptr(), st.data_ptr(), sc.data_ptr(), 1, 0)
    net.check()
    torch.cuda.synchronize()
    assert bool((st == 1).all()) and bool((x == 1).all())
    net.close()


def test_an_unaligned_input_is_refused():
    """As by the GEMM of the lift: status 1, whichever kernels serve the network."""
    from sac_b200 import fno_abi

    for F in (72, 264):
        net = _net(56, F, 1)
        x = torch.zeros(16 * 56 * F + 1, dtype=torch.bfloat16, device="cuda")[1:]
        y = torch.zeros(6, 56, F, device="cuda")
        torch.cuda.synchronize()
        for run in (net.forward, net.infer):
            with pytest.raises(fno_abi.FnoError) as e:
                run(x.data_ptr(), y.data_ptr(), 1)
            assert "status 1" in str(e.value)
        net.close()
