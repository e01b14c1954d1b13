"""The work that users of this framework have it do, as cases that can be timed.

Every case is one pass through the public Python entry points (`abi.Context`,
`batch.Batch`, `surrogate.Surrogate`, `fno_abi.Net`):

  grid   a single grid advanced from one snapshot to the next: `steps` times
         getdt + advect, then the download of w(ixG^T,nw) that a save writes;
  batch  many uneven 2D vortices set to their start on the device, advanced
         together, and gathered on the device;
  infer  one surrogate window for a set of flux tubes (Surrogate.predict);
  train  one surrogate training step over several minibatches (gradient
         accumulation), with the gradients read back for an all-reduce on the host.

Inputs are made on the GPU from the seed alone.  `exact` gives the same outputs
from plain torch in 64 bits.
"""
import math
import random

import numpy as np
import torch

from sac_b200 import abi, batch, fno_abi, params, surrogate

DEV = "cuda"
G = 2  # ghost layers per side

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
LISTED = [
    # Brio-Wu shock tube at the reference's resolution: the smallest calls, where a
    # step is launches and latency
    dict(name="shock_800", kind="grid", problem="shock", n1=800, n2=0, n3=0, fp32=False, steps=100),
    # Orszag-Tang vortex at 512^2 with keeppositive's floors in every boundary fill
    dict(name="vortex_floors_512", kind="grid", problem="vortex", n1=512, n2=512, n3=0, fp32=False, steps=30),
    # 2D flux tube, ragged size, with the Powell and resistive sources that the
    # reference's defaults and its mhdres module add
    dict(name="tube_sources_251x187", kind="grid", problem="tube", n1=251, n2=187, n3=0, fp32=False, steps=40),
    # the stratified atmosphere at the benchmark's small grid, in both storage
    # precisions, from random modes
    dict(name="atmosphere_128", kind="grid", problem="atmosphere", n1=128, n2=128, n3=128, fp32=False, steps=16),
    dict(name="atmosphere_128_fp32", kind="grid", problem="atmosphere", n1=128, n2=128, n3=128, fp32=True, steps=32),
    # the same workload at a large grid, where nothing but the device counts
    dict(name="atmosphere_256", kind="grid", problem="atmosphere", n1=256, n2=208, n3=208, fp32=False, steps=8),
    # a small ragged 3D box with every source term and open boundaries on two sides
    dict(name="box_sources_61x47x53", kind="grid", problem="box", n1=61, n2=47, n3=53, fp32=False, steps=12),
    # parameter studies: many uneven vortices at once, sizes from {64, 96, ..., 512};
    # in 32 bits sampled after every step, before the vortices' sensitivity to
    # rounding (through each instance's own dt) shows
    dict(name="batch_48", kind="batch", count=48, sizes=1, fp32=False, steps=6),
    dict(name="batch_96_fp32", kind="batch", count=96, sizes=2, fp32=True, steps=1),
    # the surrogate's roll-out: 64 samples per call, as its users run it, and a few
    # tubes on a ragged grid
    dict(name="infer_64", kind="infer", count=64, S=256, F=256),
    dict(name="infer_3_ragged", kind="infer", count=3, S=200, F=136),
    # the surrogate's training step at its minibatch
    dict(name="train_16", kind="train", count=16, S=256, F=256, minibatches=6),
]


def listed():
    return [dict(c) for c in LISTED]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    kind = rng.choice(["shock", "vortex", "tube", "atmosphere", "atmosphere", "box", "batch", "infer", "train"])
    if kind == "shock":
        return dict(kind="grid", problem="shock", n1=_log(rng, 64, 4000), n2=0, n3=0, fp32=False,
                    steps=rng.randint(20, 100))
    if kind in ("vortex", "tube"):
        return dict(kind="grid", problem=kind, n1=_log(rng, 48, 640), n2=_log(rng, 48, 640), n3=0,
                    fp32=kind == "tube" and rng.random() < 0.4, steps=rng.randint(8, 30))
    if kind == "atmosphere":
        return dict(kind="grid", problem="atmosphere", n1=_log(rng, 40, 240), n2=_log(rng, 40, 160),
                    n3=_log(rng, 40, 160), fp32=rng.random() < 0.5, steps=rng.randint(4, 10))
    if kind == "box":
        return dict(kind="grid", problem="box", n1=_log(rng, 24, 96), n2=_log(rng, 24, 96), n3=_log(rng, 24, 96),
                    fp32=rng.random() < 0.3, steps=rng.randint(4, 12))
    if kind == "batch":
        fp32 = rng.random() < 0.5
        return dict(kind="batch", count=_log(rng, 8, 90), sizes=rng.randint(10, 9999), fp32=fp32,
                    steps=1 if fp32 else rng.randint(2, 6))
    S, F = 8 * rng.randint(8, 32), 8 * rng.randint(8, 32)
    if kind == "infer":
        return dict(kind="infer", count=_log(rng, 1, 64), S=S, F=F)
    return dict(kind="train", count=_log(rng, 2, 16), S=S, F=F, minibatches=rng.randint(2, 6))


# ---------------------------------------------------------------------------
# single grids: initial states on the GPU.  Tensors are (iw, i3, i2, i1), the
# reference's Fortran order w(i1,i2,i3,iw) read from its slowest index.
# ---------------------------------------------------------------------------
class Grid:
    """Shape, coordinates, parameters, boundary types and initial state of a case."""

    def __init__(self, case, seed):
        self.gen = torch.Generator(DEV)
        self.gen.manual_seed(int(seed))
        self.host = random.Random(int(seed))
        self.n = [case[k] for k in ("n1", "n2", "n3") if case[k]]
        self.nd = len(self.n)
        self.nr = 3 if self.nd == 3 else 2
        self.np_, self.nw = 2 * self.nr + 2, 3 * self.nr + 4
        self.E = self.nr + 1
        self.shape = tuple(v + 2 * G for v in reversed(self.n))
        self.w = torch.zeros((self.nw,) + self.shape, dtype=torch.float64, device=DEV)
        self.opt = dict(gamma=5.0 / 3.0, nu=1.0, courantpar=0.8, typeadvance="fourstep",
                        precision=params.PREC_FP32 if case["fp32"] else params.PREC_FP64)
        self.restart = True  # every pass starts from the initial state
        getattr(self, case["problem"])()

    def axes(self, lows, highs):
        self.lows, self.width = lows, [(b - a) / n for n, a, b in zip(self.n, lows, highs)]
        ax = [a + (torch.arange(-G, n + G, dtype=torch.float64, device=DEV) + 0.5) * d
              for a, n, d in zip(lows, self.n, self.width)]
        self.x = torch.stack([ax[d].view([-1 if self.nd - 1 - d == k else 1 for k in range(self.nd)])
                              .expand(self.shape) for d in range(self.nd)])
        return [self.x[d] for d in range(self.nd)]

    def uniform(self, lo, hi):
        return self.host.uniform(lo, hi)

    def modes(self, amp, count, kmax):
        """Seeded random Fourier modes in rho', v and a divergence-free b', with the
        thermal pressure kept: e' gains the kinetic and magnetic energy."""
        w, nd, nr, E = self.w, self.nd, self.nr, self.E
        rnd = lambda *s: torch.randn(*s, generator=self.gen, dtype=torch.float64, device=DEV)  # noqa: E731
        k = torch.randint(-kmax, kmax + 1, (count, nd), generator=self.gen, device=DEV).double()
        k[:, 0] += (k.abs().sum(1) == 0)
        L = [d * n for d, n in zip(self.width, self.n)]
        kk = torch.zeros(count, nr, dtype=torch.float64, device=DEV)
        kk[:, :nd] = k / torch.tensor(L, dtype=torch.float64, device=DEV)
        ab = rnd(count, nr)
        ab = ab - kk * ((ab * kk).sum(1) / (kk * kk).sum(1))[:, None]
        coef = torch.cat([torch.ones(count, 1, dtype=torch.float64, device=DEV), rnd(count, nr), ab], 1)
        ph = torch.rand(count, 3, generator=self.gen, dtype=torch.float64, device=DEV) * 2 * math.pi
        ph = torch.cat([ph[:, :1], ph[:, 1:2].expand(-1, nr), ph[:, 2:].expand(-1, nr)], 1)
        C = torch.polar(coef.abs(), ph + math.pi * (coef < 0))
        ex = []
        for d in range(nd):
            a = self.x[d].reshape(-1)[:: math.prod(self.shape[nd - d:])][: self.n[d] + 2 * G]
            ex.append(torch.exp(2j * math.pi * k[:, d, None] * a[None, :] / L[d]))
        for f in range(C.shape[1]):
            lead = C[:, f, None]
            for d in range(nd - 1, 0, -1):
                lead = (lead[:, :, None] * ex[d][:, None, :]).reshape(count, -1)
            q = (lead.T @ ex[0]).imag.reshape(self.shape)
            q = amp * q / q.abs().max()
            if f == 0:
                w[0] += q * w[E + nr + 2]
            elif f <= nr:
                w[f] += (w[0] + w[E + nr + 2]) * q
            else:
                w[E + f - nr] += q
        self.energy()

    def energy(self):
        w, nr, E = self.w, self.nr, self.E
        m2 = (w[1:1 + nr] ** 2).sum(0)
        b, bg = w[E + 1:E + 1 + nr], w[E + nr + 3:]
        w[E] += 0.5 * m2 / (w[0] + w[E + nr + 2]) + 0.5 * (b * b).sum(0) + (b * bg).sum(0)

    def types(self, *per_dim):
        self.bc = [t for d in per_dim for t in (d if isinstance(d, tuple) else (d, d))]

    # -- the problems ----------------------------------------------------------
    def shock(self):
        (x,) = self.axes((0.0,), (1.0,))
        w, right = self.w, torch.arange(-G, self.n[0] + G, device=DEV) >= self.n[0] // 2
        rho, p, b2 = self.uniform(0.11, 0.14), self.uniform(0.09, 0.11), -self.uniform(0.9, 1.1)
        sel = lambda a, b: torch.where(right, torch.full_like(x, b), torch.full_like(x, a))  # noqa: E731
        w[0] = sel(1.0, rho)
        w[self.E + 1], w[self.E + 2] = 0.75, sel(1.0, b2)
        self.opt["gamma"] = 2.0
        w[self.E] = sel(1.0, p)
        self.energy()
        self.opt.update(user=params.USR_GRAVVISC)
        self.types("cont")

    def vortex(self):
        x, y = self.axes((0.0, 0.0), (1.0, 1.0))
        w, g = self.w, self.opt["gamma"]
        px, py = self.uniform(0, 1), self.uniform(0, 1)
        p = self.uniform(0.45, 0.6)
        w[0] = g * g
        w[1], w[2] = -g * g * torch.sin(2 * math.pi * (y + py)), g * g * torch.sin(2 * math.pi * (x + px))
        w[4], w[5] = -torch.sin(2 * math.pi * (y + py)), torch.sin(4 * math.pi * (x + px))
        w[3] = p / (g - 1)
        self.energy()
        self.opt.update(user=params.USR_GRAVVISC, smallfix=1, smallp=0.5, smallrho=2.75, vacuumrho=2.75)
        self.types("periodic", "periodic")

    def tube(self):
        z, xh = self.axes((0.0, -1.0), (2.0, 1.0))
        w, g, H = self.w, self.opt["gamma"], 0.3
        rhob = 100.0 * torch.exp(-z / H)
        bz = 0.5 * torch.exp(-(xh * xh) / 0.04)
        w[7], w[8] = rhob, bz
        w[6] = (H * rhob + 0.5 * (0.25 - bz * bz)) / (g - 1) + 0.5 * bz * bz
        self.modes(1e-3, 32, 8)
        om = math.sqrt(g * H) / (2 * H) * self.uniform(0.8, 1.5)
        self.drive = [10 ** self.uniform(-3.5, -2.5), om, 0.1, 0.05, 0.0, 0.1]
        self.opt.update(user=params.USR_TUBE, grav=(-1.0, 0.0, 0.0), userpar=self.drive, eta=1e-4, divbfix=1)
        self.types("cont", "periodic")

    def atmosphere(self):
        z = self.axes((0.0, 0.0, 0.0), (1.5, 1.0, 1.0))[0]
        w, g, H, B0 = self.w, self.opt["gamma"], 0.3, 0.3
        rhob = torch.exp(-z / H)
        w[9], w[10] = rhob, B0
        w[8] = rhob * H / (g - 1) + 0.5 * B0 * B0
        self.modes(1e-4, 64, 16)
        self.drive = [1e-3 * math.sqrt(g * H), 2 * math.pi / 0.3, 0.5, 0.5, 0.05, 0.1, 0.05]
        self.opt.update(user=params.USR_STRAT, grav=(-1.0, 0.0, 0.0), userpar=self.drive)
        self.types(("fixed", "cont"), "periodic", "periodic")
        self.restart = False  # a long run goes on from where it is

    def box(self):
        z = self.axes((0.0, 0.1, 0.2), (1.0, 1.25, 1.5))[0]
        w, g = self.w, self.opt["gamma"]
        w[9] = 1.0 + 0.5 * torch.exp(-z)
        for c in range(3):
            w[10 + c] = 0.3 - 0.1 * c + 0.05 * torch.sin(1.0 + c + z)
        w[8] = 0.8 * w[9] / (g - 1) + 0.5 * (w[10:13] ** 2).sum(0)
        self.modes(0.05, 12, 3)
        w[:8] += 1e-3 * torch.randn(w[:8].shape, generator=self.gen, dtype=torch.float64, device=DEV)
        self.opt.update(user=params.USR_GRAVVISC, grav=(-0.7, 0.3, 0.2), courantpar=0.4, eta=1e-3, divbfix=1)
        self.types("cont", "periodic", "cont")


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _fortran(t):
    """A host tensor (iw, i3, i2, i1) as the Fortran-order array w(i1,i2,i3,iw)."""
    return t.numpy().T


def _prepare_grid(case, seed):
    g = Grid(case, seed)
    ctx = abi.Context(params.make_params(**g.opt))
    ixM = [G + 1] * g.nd + [1] * (3 - g.nd) + [n + G for n in g.n] + [1] * (3 - g.nd)
    ctx.set_grid(g.nd, g.nr, [n + 2 * G for n in g.n], ixM, _fortran(g.x.cpu()))
    ctx.set_boundaries(params.pack_typeB([[t] * g.nw for t in g.bc]), 2 * g.nd)
    w0 = _pinned(g.w)
    ctx.upload(_fortran(w0))
    ctx.getboundary(0.0)
    st = dict(kind="grid", ctx=ctx, t=0.0, it=0, out=_pinned(g.w), steps=case["steps"], fp32=case["fp32"],
              w0=w0 if g.restart else None)
    return st


def _run_grid(s):
    ctx = s["ctx"]
    if s["w0"] is not None:  # this run starts from its initial snapshot
        ctx.upload(_fortran(s["w0"]))
        ctx.getboundary(0.0)
        s["t"], s["it"] = 0.0, 0
    for _ in range(s["steps"]):
        dt = ctx.getdt(s["it"])
        ctx.advect(dt, s["t"], s["it"])
        s["t"] += dt
        s["it"] += 1
    ctx.download(_fortran(s["out"]))
    # a run in 32 bits is saved in 32 bits
    return s["out"].to(torch.float32) if s["fp32"] else s["out"]


# ---------------------------------------------------------------------------
# batches
# ---------------------------------------------------------------------------
def _vortices(case, seed):
    nx = batch.ot_sizes(case["count"], seed=case["sizes"])
    rng = random.Random(int(seed))
    return batch.OTBatch(case["count"], nx=nx, betas=[rng.uniform(0.5, 10.0) for _ in nx])


def _prepare_batch(case, seed):
    dt = torch.float32 if case["fp32"] else torch.float64
    b = _vortices(case, seed).make(batch.ot_params(precision=params.PREC_FP32 if case["fp32"] else params.PREC_FP64))
    b.tune()
    code = "f32" if case["fp32"] else "f64"
    start = torch.empty(b.packed_size, dtype=dt, device=DEV)
    out = torch.empty_like(start)
    torch.cuda.synchronize()
    b.gather(start.data_ptr(), code)
    b.synchronize()
    return dict(kind="batch", b=b, start=start, out=out, code=code, steps=case["steps"])


def _run_batch(s):
    b = s["b"]
    b.scatter(s["start"].data_ptr(), s["code"])  # the instances at their start
    b.getboundary()
    b.advance(s["steps"])
    b.gather(s["out"].data_ptr(), s["code"])
    return s["out"]


# ---------------------------------------------------------------------------
# the surrogate
# ---------------------------------------------------------------------------
WIDTH, LAYERS, HIDDEN, CIN, COUT, MODES, NFEAT = 32, 4, 128, 16, 6, 24, 4


def _theta(seed):
    """Seeded FP32 parameters in the library's layout (groups padded to 8 values):
    the flat vector and the named groups."""
    g = torch.Generator(DEV)
    g.manual_seed(int(seed) + 17)
    nm = 2 * MODES * MODES * WIDTH * WIDTH
    bl = 1 / math.sqrt(WIDTH)
    groups = [("P", WIDTH * CIN, 1 / math.sqrt(CIN)), ("Pb", WIDTH, 1 / math.sqrt(CIN))]
    for l in range(LAYERS):
        groups += [(f"W{l}", WIDTH * WIDTH, bl), (f"Wb{l}", WIDTH, bl), (f"Rr{l}", nm, 1 / WIDTH ** 2),
                   (f"Ri{l}", nm, 1 / WIDTH ** 2)]
    bh = 1 / math.sqrt(HIDDEN)
    groups += [("Q1", HIDDEN * WIDTH, bl), ("Q1b", HIDDEN, bl), ("Q2", 8 * HIDDEN, bh), ("Q2b", 8, bh)]
    parts, named = [], {}
    for name, n, b in groups:
        p = (torch.rand(n, generator=g, device=DEV) * 2 - 1) * b
        if name == "Q2":
            p[COUT * HIDDEN:] = 0  # the rows past cout
        if name == "Q2b":
            p[COUT:] = 0
        named[name] = p
        parts.append(p)
    return torch.cat(parts), named


def _smooth(gen, count, channels, S, F):
    """Smooth random fields: a few low Fourier modes per sample and channel."""
    z = torch.randn(count, channels, 8, 8, 2, generator=gen, device=DEV)
    spec = torch.zeros(count, channels, S, F // 2 + 1, dtype=torch.complex64, device=DEV)
    spec[:, :, :8, :8] = torch.view_as_complex(z)
    q = torch.fft.irfft2(spec, s=(S, F))
    return q / q.pow(2).mean(dim=(2, 3), keepdim=True).sqrt()


SX = [0.02, 0.015, 0.03, 0.01, 0.004, 0.006]  # channel scales of the states ...
SD = [0.1 * v for v in SX]                    # ... and of their change in a window


def _tubes(case, seed):
    """The raw perturbations of `count` flux tubes and their drivers."""
    gen = torch.Generator(DEV)
    gen.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    n = case["count"]
    A, om = 10 ** rng.uniform(-3.5, -2.5, n), rng.uniform(0.9, 1.6, n)
    st = _smooth(gen, n, COUT, case["S"], case["F"]) * torch.tensor(SX, device=DEV).view(1, -1, 1, 1)
    return (st * torch.tensor(A, dtype=torch.float32, device=DEV).view(-1, 1, 1, 1)).contiguous(), A, om


def _prepare_infer(case, seed):
    state, A, om = _tubes(case, seed)
    sur = surrogate.Surrogate(S=case["S"], F=case["F"], batch=1, infer_batch=min(64, case["count"]), seed=None)
    sur.net.set_params(_theta(seed)[0].cpu().numpy())
    sur.set_scales(SX, SD)
    torch.cuda.synchronize()
    return dict(kind="infer", sur=sur, start=state, state=state.clone(), A=A, om=om, t=0.7)


def _run_infer(s):
    with torch.cuda.stream(s["sur"].stream):
        s["state"].copy_(s["start"])
    s["sur"].predict(s["state"], s["A"], s["om"], s["t"])
    return s["state"]


def _minibatches(case, seed):
    gen = torch.Generator(DEV)
    gen.manual_seed(int(seed))
    out = []
    for _ in range(case["minibatches"]):
        x = _smooth(gen, case["count"], CIN, case["S"], case["F"]).to(torch.bfloat16)
        t = _smooth(gen, case["count"], COUT, case["S"], case["F"]).to(torch.bfloat16)
        out.append((x, t))
    return out


def _prepare_train(case, seed):
    B, S, F = case["count"], case["S"], case["F"]
    net = fno_abi.Net(S=S, F=F, width=WIDTH, layers=LAYERS, hidden=HIDDEN, cin=CIN, cout=COUT, max_batch=B, seed=None)
    net.set_params(_theta(seed)[0].cpu().numpy())
    st = dict(kind="train", net=net, data=_minibatches(case, seed), B=B,
              y=torch.empty(B, COUT, S, F, device=DEV),
              dy=torch.zeros(B, net.cpad, S, F, dtype=torch.bfloat16, device=DEV),
              loss=torch.zeros(1, device=DEV), stream=torch.cuda.ExternalStream(net.stream))
    torch.cuda.synchronize()
    return st


def _run_train(s):
    net, B = s["net"], s["B"]
    with torch.cuda.stream(s["stream"]):
        s["loss"].zero_()
    net.zero_grad()
    for x, t in s["data"]:
        net.forward(x.data_ptr(), s["y"].data_ptr(), B)
        net.mse(s["y"].data_ptr(), t.data_ptr(), s["dy"].data_ptr(), s["loss"].data_ptr(), B)
        net.backward(s["dy"].data_ptr())
    # the ranks of a training job exchange their gradients in the weights' 16 bits
    return s["loss"], torch.from_numpy(net.get_grads()).to(torch.bfloat16)


def prepare(case, seed):
    return dict(grid=_prepare_grid, batch=_prepare_batch, infer=_prepare_infer, train=_prepare_train)[case["kind"]](
        case, seed)


def run(state):
    return dict(grid=_run_grid, batch=_run_batch, infer=_run_infer, train=_run_train)[state["kind"]](state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(nd, nr, cells, size):
    """One RK4 step with its getdt.  Bytes: the advanced variables and the
    background of a stage are read once and the result written once, in the four
    stages and the two combinations of the scheme (14 passes over the variables, 4
    over the background).  Operations: fluxes and their gradients, setnu's
    quotients, the hyperdiffusion terms."""
    NP, NB, NR = 2 * nr + 2, nr + 2, 2 * nd + nd * nd + nd * (nd - 1)
    nbytes = cells * (14 * NP * size + 4 * NB * 8)
    per_stage = 40 * nr + nd * (8 * nr + 30) + 7 * (nd * NP + nd * nd) + 28 * NR + 24 * nd * nd + 62 * nd * (nd - 1)
    return nbytes, cells * 4 * per_stage


def _net_work(case, n):
    S, F = case["S"], case["F"]
    P, J, R = S * F, 2 * MODES, 4 * MODES
    layer = 2 * WIDTH * S * F * J * 2 + 2 * WIDTH * J * S * R * 2 + 16 * MODES * MODES * WIDTH * WIDTH + 2 * P * WIDTH ** 2
    return n * (2 * P * CIN * WIDTH + LAYERS * layer + 2 * P * HIDDEN * (WIDTH + COUT))


def work(case):
    if case["kind"] == "grid":
        n = [case[k] for k in ("n1", "n2", "n3") if case[k]]
        nd, nr = len(n), 3 if len(n) == 3 else 2
        full = math.prod(v + 2 * G for v in n) * (3 * nr + 4) * (4 if case["fp32"] else 8)
        b, f = _step_work(nd, nr, math.prod(n), 4 if case["fp32"] else 8)
        return {"bytes": case["steps"] * b + full, "flops": case["steps"] * f}
    if case["kind"] == "batch":
        size = 4 if case["fp32"] else 8
        cells = sum(a * b for a, b in batch.ot_sizes(case["count"], seed=case["sizes"]))
        b, f = _step_work(2, 2, cells, size)
        return {"bytes": case["steps"] * b + 2 * cells * 6 * size, "flops": case["steps"] * f}
    P, weights = case["S"] * case["F"], 2 * LAYERS * 2 * MODES * MODES * WIDTH * WIDTH
    if case["kind"] == "infer":
        return {"bytes": case["count"] * P * COUT * 8 + 2 * weights, "flops": _net_work(case, case["count"])}
    n = case["count"] * case["minibatches"]
    return {"bytes": n * P * (CIN + COUT) * 2 + weights * (2 + 4), "flops": 3 * _net_work(case, n)}


# ---------------------------------------------------------------------------
# the same in 64 bits: the MHD scheme on whole arrays
# ---------------------------------------------------------------------------
class Scheme:
    """The perturbed-MHD scheme (centdiff4, gravity, hyperdiffusion, driver,
    resistive and Powell sources, fills, RK4, getdt) for one grid."""

    def __init__(self, n, x, bc, opt):
        self.n, self.nd, self.bc, self.opt = n, len(n), bc, opt
        self.nr = 3 if self.nd == 3 else 2
        self.E = self.nr + 1
        self.gam = opt["gamma"]
        self.grav = list(opt.get("grav", (0.0, 0.0, 0.0)))
        # a Cartesian grid: the width of dimension d varies along d alone
        self.dx = []
        for d in range(self.nd):
            a = x[d].movedim(self.ax(d), 0).reshape(n[d] + 2 * G, -1)[:, 0]
            lo = a[G] - 3 * (a[G + 1] - a[G]), a[G + n[d] - 1] + 3 * (a[G + n[d] - 1] - a[G + n[d] - 2])
            e = torch.cat([lo[0][None], a, lo[1][None]])
            self.dx.append((0.5 * (e[2:] - e[:-2])).view([-1 if k == self.ax(d) else 1 for k in range(-self.nd, 0)]))
        self.mesh = tuple([slice(G, G + v) for v in reversed(n)])
        self.inside = torch.zeros([v + 2 * G for v in reversed(n)], dtype=torch.bool, device=x.device)
        self.inside[self.mesh] = True
        self.keep4, self.keep1 = [], []
        for d in range(self.nd):
            p = torch.arange(-G, n[d] + G, device=x.device)
            view = [-1 if k == self.ax(d) else 1 for k in range(-self.nd, 0)]
            self.keep4.append(((p >= 2) & (p < n[d] - 2)).double().view(view))
            k1 = torch.ones_like(p, dtype=torch.bool)
            if bc[2 * d] != "periodic":
                k1 &= p > 0
            if bc[2 * d + 1] != "periodic":
                k1 &= p < n[d] - 1
            self.keep1.append(k1.double().view(view))
        up, user = opt.get("userpar"), opt["user"]
        self.prof = None
        if user == params.USR_STRAT:
            self.prof = torch.exp(-((x[1] - up[2]) ** 2 + (x[2] - up[3]) ** 2) / up[4] ** 2) * torch.exp(
                -(x[0] - up[5]) ** 2 / up[6] ** 2)
        elif user == params.USR_TUBE:
            self.prof = torch.exp(-(x[0] - up[2]) ** 2 / up[3] ** 2) * torch.exp(-(x[1] - up[4]) ** 2 / up[5] ** 2)
        self.comp = 1 if user == params.USR_STRAT else 2
        self.maxnu, self.fix, self.it0, self.dtdiff = 0.0, None, None, 0.5

    @staticmethod
    def ax(d):
        return -(d + 1)

    def sh(self, q, d, k):
        return torch.roll(q, -k, self.ax(d))

    def g4(self, q, d):
        s = self.sh
        return self.keep4[d] * -(s(q, d, 2) - 8 * (s(q, d, 1) - s(q, d, -1)) - s(q, d, -2)) / self.dx[d] / 12

    def g1(self, q, d):
        return self.keep1[d] * (self.sh(q, d, 1) - self.sh(q, d, -1)) / self.dx[d] / 2

    def speeds(self, w):
        nr, E, g = self.nr, self.E, self.gam
        m, b, bg = w[1:1 + nr], w[E + 1:E + 1 + nr], w[E + nr + 3:]
        rt = w[0] + w[E + nr + 2]
        p = (g - 1) * (w[E] - 0.5 * (m * m).sum(0) / rt - 0.5 * (b * b).sum(0) - (b * bg).sum(0))
        cs2 = g * (p + (g - 1) * (w[E + nr + 1] - 0.5 * (bg * bg).sum(0))) / rt
        cf2 = ((b + bg) ** 2).sum(0) / rt + cs2
        return [torch.sqrt(0.5 * (cf2 + torch.sqrt(cf2 * cf2 - 4 * cs2 * (b[d] + bg[d]) ** 2 / rt))) + (m[d] / rt).abs()
                for d in range(self.nd)]

    def nu(self, q, d, scale):
        """setnu's coefficients at the two faces of every cell (0 outside the mesh)."""
        n, a = self.n[d], self.ax(d)
        t = torch.cat([q.narrow(a, G + 3, 1), q, q.narrow(a, G + n - 4, 1)], a)
        L = t.shape[a]
        d1 = (t.narrow(a, 1, L - 1) - t.narrow(a, 0, L - 1)).abs()
        d3 = (3 * (t.narrow(a, 2, L - 3) - t.narrow(a, 1, L - 3)) - (t.narrow(a, 3, L - 3) - t.narrow(a, 0, L - 3))).abs()
        # faces i-1/2 of the mesh cells and the last one's right face: n + 1 of them
        m1 = torch.stack([d1.narrow(a, k, n + 1) for k in range(5)]).amax(0)
        m3 = torch.stack([d3.narrow(a, k, n + 1) for k in range(3)]).amax(0)
        r = torch.where(m1 > 0, scale * m3 / torch.where(m1 > 0, m1, torch.ones_like(m1)), torch.zeros_like(m1))
        nl, nr = torch.zeros_like(q), torch.zeros_like(q)
        nl.narrow(a, G, n).copy_(r.narrow(a, 0, n))
        nr.narrow(a, G, n).copy_(r.narrow(a, 1, n))
        nl, nr = nl * self.dx[d] * self.inside, nr * self.dx[d] * self.inside
        self.maxnu = torch.maximum(torch.as_tensor(self.maxnu, device=q.device), torch.maximum(nl.max(), nr.max()))
        return nl, nr

    def rate(self, w, base, qdt, t):
        """base + qdt (flux divergence and sources of w), valid on the mesh."""
        nd, nr, E, g = self.nd, self.nr, self.E, self.gam
        m, b, bg = w[1:1 + nr], w[E + 1:E + 1 + nr], w[E + nr + 3:]
        eb, rhob = w[E + nr + 1], w[E + nr + 2]
        rt = w[0] + rhob
        v = m / rt
        new = base[:E + 1 + nr].clone()
        b2, m2, bb = (b * b).sum(0), (m * m).sum(0), (b * bg).sum(0)
        pt = (g - 1) * (w[E] - 0.5 * m2 / rt) - (g - 2) * (bb + 0.5 * b2)
        s1, s2 = (bg * m).sum(0), (b * m).sum(0)
        fb = (g - 1) * eb - 0.5 * (g - 2) * (bg * bg).sum(0)
        for d in range(nd):
            new[0] -= qdt * self.g4(rhob * v[d] + v[d] * w[0], d)
            for c in range(nr):
                f = -(b[c] * bg[d] + b[d] * bg[c]) - b[c] * b[d] + v[d] * m[c]
                new[1 + c] -= qdt * self.g4(f + pt if c == d else f, d)
                if c != d:
                    new[E + 1 + c] -= qdt * self.g4(v[d] * (b[c] + bg[c]) - v[c] * (b[d] + bg[d]), d)
            fe = (m[d] * pt - b[d] * s1 - bg[d] * s2) / rt + eb * v[d] - b[d] * s2 / rt + v[d] * w[E]
            new[E] -= qdt * (self.g4(fe, d) + self.g4(v[d], d) * fb)
            for k in range(nd):
                new[E] += qdt * bg[k] * bg[d] * self.g4(v[d], k)
        for d in range(nd):
            if self.grav[d]:
                new[1 + d] += qdt * self.grav[d] * w[0]
                new[E] += qdt * self.grav[d] * w[0] * v[d]
        self.viscous(w, new, qdt, rt, m, b, v, b2, m2)
        if self.prof is not None:
            vel = self.opt["userpar"][0] * math.sin(self.opt["userpar"][1] * t) * self.prof
            r = new[0] + rhob
            new[self.comp] += r * vel * qdt
            new[E] += r * vel * vel * qdt / 2
        B, eta = b + bg, self.opt.get("eta", 0.0)
        if eta:
            self.resist(new, B, eta * qdt)
        if self.opt.get("divbfix") and nd > 1:
            div = qdt * sum(self.g4(B[d], d) for d in range(nd))
            new[1:1 + nr] -= B * div
            new[E + 1:E + 1 + nr] -= v * div
            new[E] -= (v * B).sum(0) * div
        return new

    def viscous(self, w, new, qdt, rt, m, b, v, b2, m2):
        nd, E, sh, dx = self.nd, self.E, self.sh, self.dx
        ct = [c[self.mesh].max() for c in self.speeds(w)]
        half = lambda q, d, k: 0.5 * (q + sh(q, d, k))  # noqa: E731
        q173 = w[E] - 0.5 * (b2 + m2 / rt)
        left = lambda q, d: self.keep1[d] * (q - sh(q, d, -1)) / dx[d]  # noqa: E731
        right = lambda q, d: self.keep1[d] * (sh(q, d, 1) - q) / dx[d]  # noqa: E731
        for tgt, q in ((0, w[0]), (E, q173)):
            for k in range(nd):
                nl, nr = self.nu(q, k, ct[k] * 0.04)
                new[tgt] += qdt * (nr * right(q, k) - nl * left(q, k)) / dx[k]
        for k in range(nd):
            rL, rR = half(rt, k, -1), half(rt, k, 1)
            for l in range(nd):
                nl, nr = self.nu(v[l], k, ct[k] * 0.4)
                tL, tR = nl * left(v[l], k), nr * right(v[l], k)
                twice = 2 if l == k else 1
                new[1 + l] += twice * qdt * (rR * tR - rL * tL) / dx[k] / 2
                new[E] += twice * qdt * (half(m[l], k, 1) * tR - half(m[l], k, -1) * tL) / dx[k] / 2
                if l != k:
                    H = self.g1(v[l], k) * (nl + nr) / 4
                    new[1 + k] += qdt * self.g1(rt * H, l)
                    new[E] += qdt * self.g1(m[k] * H, l)
        for k in range(nd):
            for l in range(nd):
                if l == k:
                    continue
                nl, nr = self.nu(b[l], k, ct[k] * 0.04)
                K = self.g1(b[l], k) * (nl + nr) / 2
                new[E + 1 + k] -= qdt * self.g1(K, l)
                new[E] -= qdt * self.g1(K * b[k], l)
                tL, tR = nl * left(b[l], k), nr * right(b[l], k)
                new[E + 1 + l] += qdt * (tR - tL) / dx[k]
                new[E] += qdt * (tR * half(b[l], k, 1) - tL * half(b[l], k, -1)) / dx[k]

    def resist(self, new, B, eq):
        """qdt eta (-curl J) into b and div (B x J) into e, central differences."""
        nd, nr, E = self.nd, self.nr, self.E
        lv = lambda i, j, k: (i - j) * (j - k) * (k - i) // 2  # noqa: E731
        c1 = lambda q, d: (self.sh(q, d, 1) - self.sh(q, d, -1)) / self.dx[d] / 2  # noqa: E731
        J = [sum((lv(i, j, k) * c1(B[k], j) for j in range(nd) for k in range(nr) if lv(i, j, k)),
                 torch.zeros_like(B[0])) for i in range(3)]
        for d in range(nd):
            for i in range(nr):
                for k in range(3):
                    if lv(i, d, k):
                        new[E + 1 + i] -= lv(i, d, k) * c1(J[k], d) * eq
            for j in range(nr):
                for k in range(3):
                    if lv(d, j, k):
                        new[E] += lv(d, j, k) * c1(B[j] * J[k], d) * eq

    def fill(self, w):
        if self.opt.get("smallfix"):
            self.floors(w)
        for d in range(self.nd):
            n, a = self.n[d], self.ax(d)
            for up in (0, 1):
                kind, at = self.bc[2 * d + up], (G + n if up else 0)
                if kind == "periodic":
                    w.narrow(a, at, G).copy_(w.narrow(a, G if up else n, G).clone())
                elif kind == "cont" or self.fix is None:  # the first fill of a fixed side copies the edge
                    w.narrow(a, at, G).copy_(w.narrow(a, G + n - 1 if up else G, 1).clone().expand(
                        w.narrow(a, at, G).shape))
                else:  # fixed: what the first fill left there
                    w.narrow(a, at, G).copy_(self.fix.narrow(a, at, G)[: w.shape[0]])
        if self.fix is None:
            self.fix = w.clone()

    def floors(self, full):
        """keeppositive: the vacuum state below smallrho, then the energy rebuilt from
        the floored pressure where any pressure is low."""
        o, nr, E, g = self.opt, self.nr, self.E, self.gam
        w = full[(slice(None),) + self.mesh]
        m, b, bg = w[1:1 + nr], w[E + 1:E + 1 + nr], w[E + nr + 3:]
        eb, rhob = w[E + nr + 1], w[E + nr + 2]
        b2 = (b * b).sum(0)
        vac = w[0] + rhob < o["smallrho"]
        m.mul_(~vac)
        w[0].copy_(torch.where(vac, o["vacuumrho"] - rhob, w[0]))
        w[E].copy_(torch.where(vac, o["smallp"] / (g - 1) + 0.5 * b2 - eb, w[E]))
        m2 = (m * m).sum(0)
        p = (g - 1) * (w[E] - 0.5 * m2 / (w[0] + rhob) - 0.5 * b2 - (b * bg).sum(0))
        if bool((p < max(0.0, o["smallp"])).any()) and o["smallp"] > 0:
            w[E].copy_(p.clamp_min(o["smallp"]) / (g - 1) + 0.5 * (m2 / w[0] + b2) - eb)

    def advect1(self, qdt, t, wct, base):
        out = base.clone()
        sel = (slice(None, self.E + 1 + self.nr),) + self.mesh
        out[sel] = self.rate(wct, base, qdt, t)[(slice(None),) + self.mesh]
        self.fill(out)
        return out

    def step(self, w, dt, t):
        w1 = self.advect1(dt / 2, t, w, w)
        w2 = self.advect1(dt / 2, t, w1, w)
        w3 = self.advect1(dt, t, w2, w)
        np_ = self.E + 1 + self.nr
        acc = (w1[:np_] + 2 * w2[:np_] + w3[:np_] - 4 * w[:np_]) / 3
        out = self.advect1(dt / 6, t, w3, w)
        out[:np_] += acc
        return out

    def getdt(self, w, it):
        dx = [d.narrow(self.ax(k), G, self.n[k]) for k, d in enumerate(self.dx)]
        sp = [c[self.mesh] / dx[k] for k, c in enumerate(self.speeds(w))]
        dt = self.opt["courantpar"] / float(torch.stack([c.max() for c in sp]).max())
        dmin = [float(d.min()) for d in dx]
        if self.opt.get("eta", 0.0):
            dt = min(dt, self.dtdiff * min(dmin) ** 2 / self.opt["eta"])
        self.dtdiff = 0.25
        nu, self.maxnu = float(self.maxnu), 0.0
        if nu > 0:
            dt = min([dt] + [0.25 * d * d / nu for d in dmin])
        if self.it0 is None:
            self.it0 = it
        for g in self.grav[: self.nd]:
            if g:
                dt = min(dt, 1 / math.sqrt(abs(g) / min(dmin)))
        return dt

    def advance(self, w, steps):
        self.fill(w)
        t = 0.0
        for k in range(steps):
            dt = self.getdt(w, k)
            w = self.step(w, dt, t)
            t += dt
        return w


def _fno64(th, x, S, F):
    """The network in 64 bits (autograd works through it)."""
    c = math.sqrt(2 / math.pi)
    gelu = lambda z: 0.5 * z * (1 + torch.tanh(c * (z + 0.044715 * z ** 3)))  # noqa: E731
    pw = lambda wt, b, z: torch.einsum("oi,bisf->bosf", wt, z) + b.view(1, -1, 1, 1)  # noqa: E731
    kx = torch.cat([torch.arange(MODES), torch.arange(S - MODES, S)]).to(x.device)
    v = pw(th["P"].view(WIDTH, CIN), th["Pb"], x)
    for l in range(LAYERS):
        R = torch.complex(th[f"Rr{l}"], th[f"Ri{l}"]).view(2 * MODES, MODES, WIDTH, WIDTH)
        U = torch.fft.rfft2(v)[:, :, kx, :MODES]
        O = torch.zeros(v.shape[0], WIDTH, S, F // 2 + 1, dtype=U.dtype, device=x.device)
        O = O.index_copy(2, kx, torch.nn.functional.pad(torch.einsum("bixy,xyio->boxy", U, R),
                                                        (0, F // 2 + 1 - MODES)))
        z = pw(th[f"W{l}"].view(WIDTH, WIDTH), th[f"Wb{l}"], v) + torch.fft.irfft2(O, s=(S, F))
        v = gelu(z) if l < LAYERS - 1 else z
    h = gelu(pw(th["Q1"].view(HIDDEN, WIDTH), th["Q1b"], v))
    return pw(th["Q2"].view(8, HIDDEN), th["Q2b"], h)[:, :COUT]


def exact(case, seed):
    if case["kind"] == "grid":
        g = Grid(case, seed)
        return Scheme(g.n, g.x, g.bc, g.opt).advance(g.w, case["steps"])
    if case["kind"] == "batch":
        vs, parts = _vortices(case, seed), []
        opt = dict(gamma=5.0 / 3.0, courantpar=0.8, user=params.USR_GRAVVISC)
        for i, n in enumerate(vs.nx):
            w = torch.from_numpy(np.ascontiguousarray(vs.state(i).T)).to(DEV)
            x = torch.from_numpy(np.ascontiguousarray(vs.x(i).T)).to(DEV)
            s = Scheme(list(n), x, ["periodic"] * 4, opt)
            w = s.advance(w, case["steps"])
            parts.append(w[(slice(0, 6),) + s.mesh].reshape(-1))
        return torch.cat(parts)
    S, F = case["S"], case["F"]
    th = {k: p.double() for k, p in _theta(seed)[1].items()}
    if case["kind"] == "infer":
        state, A, om = _tubes(case, seed)
        out, t = [], 0.7
        omega_ac = math.sqrt(5.0 / 3.0 * 0.3) / 0.6
        sx, sd = (torch.tensor(v, dtype=torch.float64, device=DEV).view(-1, 1, 1) for v in (SX, SD))
        gs = (torch.arange(S, device=DEV) / S - 0.5).double().view(1, S, 1).expand(1, S, F)
        gf = (torch.arange(F, device=DEV) / F).double().view(1, 1, F).expand(1, S, F)
        for i in range(case["count"]):
            f = [math.sin(om[i] * t), math.cos(om[i] * t), om[i] / omega_ac - 1.25, math.log10(A[i]) + 3.0]
            f = torch.tensor(f, dtype=torch.float64, device=DEV).view(NFEAT, 1, 1).expand(NFEAT, S, F)
            s = state[i].double()
            x = torch.cat([s / sx / A[i], f, gs, gf])
            x = torch.cat([x, torch.zeros(CIN - x.shape[0], S, F, dtype=x.dtype, device=DEV)])
            out.append(s + A[i] * sd * _fno64(th, x[None], S, F)[0])
        return torch.stack(out)
    loss, grads = 0.0, None
    names = list(th)
    for p in th.values():
        p.requires_grad_(True)
    for x, t in _minibatches(case, seed):
        for i in range(0, case["count"], 4):  # a few samples at a time: the tape is held in 64 bits
            y = _fno64(th, x[i:i + 4].double(), S, F)
            part = (y - t[i:i + 4].double()).pow(2).sum() / t.numel()
            got = torch.autograd.grad(part, [th[k] for k in names])
            grads = list(got) if grads is None else [a + b for a, b in zip(grads, got)]
            loss += float(part.detach())
    return torch.tensor([loss], dtype=torch.float64), torch.cat(grads).cpu()
