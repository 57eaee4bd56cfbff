"""Performance cases of the framework: what its users run, over the sizes they run it at.

A case is a simulation job (some time steps through ChannelSolver, then the
state back in the host's arrays) or a training iteration of the learned
closure (MLPClosure).  `prepare` gives what a program holds before the timed
call: the solver with its uploaded, projected start field and the pinned host
arrays the state returns to, or the network with its mini-batch.  `run`
continues from where the last pass ended, as a simulation does.

`exact` restates the step in 64 bits with plain torch operations (dense or
FFT solves where the library eliminates), independent of the library.
"""
import math

import numpy as np
import torch

from channel3d_b200 import ChannelConfig, ChannelSolver
from channel3d_b200.mlp import MLPClosure

PI = math.pi


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _job(kind, nx, ny, nz, nsteps, **kw):
    """kind: pimp, fimp (2nd order, channel), o4 (4th order, channel with
    statistics), tg (explicit, triply periodic Taylor-Green vortex), les
    (partially implicit with a subgrid model)."""
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "nsteps": nsteps, "precision": "fp64", "re": 5600.0,
         "dt": 0.001, "calls": 1, "les": 0}
    c.update(kw)
    return c


def listed():
    return [
        # smallest calls: a Fortran host that calls one step per iteration on the 64^3 channel
        dict(_job("pimp", 64, 64, 64, 20, dt=0.002, calls=20), name="channel64_host_loop"),
        # production LES with the learned closure on its 48^3 grid
        dict(_job("les", 48, 48, 48, 40, re=13750.0, dt=0.002, les=11), name="les48_learned_closure"),
        # the reference's Taylor-Green input: explicit scheme, triply periodic box
        dict(_job("tg", 64, 64, 64, 20, dt=0.01), name="taylor_green64_explicit"),
        # a ragged grid in mixed precision: odd ny, no power-of-two x or z
        dict(_job("pimp", 96, 65, 54, 20, dt=0.002, precision="mixed"), name="ragged96x65x54_mixed"),
        # 4th-order Re_tau 180 DNS with its statistics every 10 steps
        dict(_job("o4", 128, 128, 128, 20, calls=2), name="channel128_4th_stats"),
        # the same box, fully implicit (ADI) 2nd order
        dict(_job("fimp", 128, 128, 128, 20), name="channel128_adi"),
        # the 192^3 DNS that produces the learned closure's training data
        dict(_job("pimp", 192, 192, 192, 10, re=13750.0, dt=0.0005), name="channel192_fp64"),
        # Re_tau 395 DNS, both precisions
        dict(_job("pimp", 256, 192, 256, 20, re=13750.0, dt=0.0005), name="channel256x192x256_fp64"),
        dict(_job("pimp", 256, 192, 256, 20, re=13750.0, dt=0.0005, precision="mixed"), name="channel256x192x256_mixed"),
        # the large throughput run (Re_tau 590), both precisions
        dict(_job("pimp", 768, 384, 576, 10, re=21900.0, dt=0.0003), name="channel768x384x576_fp64"),
        dict(_job("pimp", 768, 384, 576, 20, re=21900.0, dt=0.0003, precision="mixed"), name="channel768x384x576_mixed"),
        # one training iteration of the closure's network: forward, backward, Adam
        {"kind": "train", "batch": 65536, "name": "closure_training65536"},
    ]


def _smooth(lo, hi, even):
    """Products of 2 and 3 in [lo, hi] (even ones only where asked)."""
    return sorted(v for a in range(12) for b in range(7) for v in [2 ** a * 3 ** b] if lo <= v <= hi and not (even and v % 2))


def _log_pick(rng, values):
    t = math.exp(rng.uniform(math.log(values[0]), math.log(values[-1])))
    return min(values, key=lambda v: abs(math.log(v / t)))


def draw(rng):
    what = rng.choices(["pimp", "mixed", "fimp", "o4", "tg", "les", "train"], [30, 30, 10, 10, 6, 8, 6])[0]
    if what == "train":
        return {"kind": "train", "batch": int(math.exp(rng.uniform(math.log(4096), math.log(65536))))}
    big = what in ("pimp", "mixed")
    while True:
        nx = _log_pick(rng, _smooth(32, 768 if big else 256, True))
        nz = _log_pick(rng, _smooth(32, 576 if big else 192, False))
        ny = int(math.exp(rng.uniform(math.log(24), math.log(384 if big else 160))))
        nsteps = rng.randint(5, 40)
        if nx * ny * nz * nsteps <= (1.5e9 if big else 1.2e8):
            break
    dt = min(0.002, 0.1 * 2 * PI / nx)
    re = rng.choice([5600.0, 13750.0])
    if what == "mixed":
        return _job("pimp", nx, ny, nz, nsteps, precision="mixed", re=re, dt=dt)
    if what == "tg":
        return _job("tg", nx, min(ny, 96), nz, nsteps, dt=min(0.01, dt * 2))
    if what == "les":
        return _job("les", nx, ny, nz, nsteps, re=13750.0, dt=dt, les=rng.choice([10, 11]))
    if what == "o4":
        return _job("o4", nx, ny, nz, nsteps, dt=dt, calls=1)
    return _job(what, nx, ny, nz, nsteps, re=re, dt=dt, calls=rng.choice([1, 1, nsteps]))


def _config(c):
    kind, ny = c["kind"], c["ny"]
    grid = dict(nxc=c["nx"], nyc=ny, nzc=c["nz"], dtMax=c["dt"], precision=c["precision"])
    if kind == "tg":
        return ChannelConfig(FlowType=3, xlx=2 * PI, yly=2 * PI, zlz=2 * PI, xnu=6.25e-4, IsImplicit=0, BcOption=[0] * 6,
                             IsUxConst=False, ubulk=0.0, ybulk1=0.0, ybulk2=2 * PI, nSection=1, SectionLength=[1.0],
                             nycSection=[ny], StretType=[0], StretOption=[0], SectioncStret=[0.0], **grid)
    box = (4 * PI, 4 * PI / 3) if kind in ("o4", "fimp") else (2 * PI, PI)
    return ChannelConfig(order=4 if kind == "o4" else 2, IsImplicit=2 if kind == "fimp" else 1, xlx=box[0], yly=2.0,
                         zlz=box[1], xnu=2.0 / c["re"], LES_type=c["les"], Cs=0.1, nSection=2,
                         SectionLength=[1.0, 1.0], nycSection=[ny // 2, ny - ny // 2], StretType=[1, 1],
                         StretOption=[0, 1], SectioncStret=[2.0, 2.0], **grid)


# ---------------------------------------------------------------------------
# inputs (torch on the GPU, from the seed alone)
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _mesh(c):
    """yp(1:nyc+1): uniform, or two tanh-stretched halves (stretch 2.0)."""
    ny = c["ny"]
    if c["kind"] == "tg":
        return 2 * PI * np.arange(ny + 1) / ny
    lo, hi, st = ny // 2, ny - ny // 2, 2.0
    low = np.tanh(st * (np.arange(lo + 1) / lo - 1.0)) / np.tanh(st) + 1.0
    up = 1.0 + np.tanh(st * (np.arange(hi + 1) / hi)) / np.tanh(st)
    yp = np.concatenate([low, up[1:]])
    yp[0], yp[lo], yp[-1] = 0.0, 1.0, 2.0
    return yp


def _start(c, yp, seed):
    """Start fields (nz, ny, nx), FP64: laminar profile with 10% noise, or the
    Taylor-Green vortex with 1% noise."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    g = _generator(seed)
    noise = lambda: torch.empty((nz, ny, nx), dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g)  # noqa: E731
    y = torch.tensor(0.5 * (yp[1:] + yp[:-1]), device="cuda")[None, :, None]
    if c["kind"] == "tg":
        x = 2 * PI / nx * torch.arange(nx, device="cuda", dtype=torch.float64)[None, None, :]
        z = 2 * PI / nz * (torch.arange(nz, device="cuda", dtype=torch.float64)[:, None, None] + 0.5)
        yn = torch.tensor(yp[:-1], device="cuda")[None, :, None]
        f = [torch.sin(x) * torch.cos(y) * torch.cos(z) + 0.01 * noise(),
             -torch.cos(x + PI / nx) * torch.sin(yn) * torch.cos(z) + 0.01 * noise(), 0.01 * noise()]
    else:
        f = [1.5 * (1.0 - (y - 1.0) ** 2) + 0.1 * noise(), 0.1 * noise(), 0.1 * noise()]
        f[1][:, 0, :] = 0.0
    return f + [torch.zeros((nz, ny, nx), dtype=torch.float64, device="cuda")]


def _closure(seed):
    """The closure's network and standardisation: parameters of its initialisation's
    size (W uniform, fan-in scaled) and wall-unit statistics of a channel."""
    rng = np.random.default_rng(seed)
    p = np.concatenate([rng.uniform(-1, 1, n) * (math.sqrt(6.0 / fan) if w else 0.1)
                        for n, fan, w in ((640, 10, 1), (64, 1, 0), (4096, 64, 1), (64, 1, 0), (4096, 64, 1), (64, 1, 0),
                                          (384, 64, 1), (6, 1, 0))]).astype(np.float32)
    n = np.zeros(52, dtype=np.float32)
    n[9], n[10:19], n[19] = 150.0, 0.5, 100.0
    n[20:30], n[30:40], n[46:52] = -30.0, 30.0, 0.1
    return p, n


def _batch(c, seed):
    g = _generator(seed)
    X = torch.randn((c["batch"], 10), device="cuda", generator=g)
    T = torch.randn((c["batch"], 6), device="cuda", generator=g)
    return X, T


# ---------------------------------------------------------------------------
# the measured path
# ---------------------------------------------------------------------------
NAMES = ("ux", "uy", "uz", "p")


def prepare(case, seed):
    if case["kind"] == "train":
        X, T = _batch(case, seed)
        return {"case": case, "net": MLPClosure(params=_closure(seed)[0]), "X": X, "T": T}
    yp = _mesh(case)
    s = ChannelSolver(_config(case), yp=yp)
    shape = (case["nz"], case["ny"], case["nx"])
    out = {}
    for k, f in zip(NAMES, _start(case, yp, seed)):
        host = torch.empty(shape, dtype=torch.float64, pin_memory=True)
        host.copy_(f)
        out[k] = host.numpy()
    s.upload(*(out[k] for k in NAMES))
    s.project()
    if case["les"] == 11:
        s.sgs_mlp_set(*_closure(seed))
    return {"case": case, "solver": s, "out": out}


def run(state):
    c = state["case"]
    if c["kind"] == "train":
        net = state["net"]
        loss = net.grad(state["X"], state["T"])
        net.adam(1e-3)
        return {"loss": loss, "grad": net.g, "params": net.P}
    s = state["solver"]
    r = {}
    for _ in range(c["calls"]):
        s.step(c["nsteps"] // c["calls"])
        if c["kind"] == "o4":
            s.stats_accumulate()
    if c["kind"] == "o4":
        r["stat"] = s.stats_fetch(reset=True)[0]
    r.update(s.download(out=state["out"]))
    return r


def work(case):
    """Full-field arrays that the data dependencies of a substep make cross the
    memory once: right-hand side and elimination 13 (u, v, w, p, three histories
    in; histories and eliminated values out), divergence with its x and z
    transform 4, y solves 2, inverse transforms 2, projection 9."""
    if case["kind"] == "train":
        b = case["batch"]
        return {"bytes": b * 64.0 + 9414 * 4 * 8.0, "flops": 3 * 2 * (640 + 4096 + 4096 + 384) * float(b)}
    n = float(case["nx"] * case["ny"] * case["nz"])
    steps = case["nsteps"] // case["calls"] * case["calls"]
    word = 4 if case["precision"] == "mixed" else 8
    arrays = 90 + {"fimp": 36, "les": 30 if case["les"] == 11 else 16}.get(case["kind"], 0)
    flops = 3 * (200 + 5 * math.log2(case["nx"] * case["nz"]))
    if case["kind"] == "o4":
        flops *= 1.5
    if case["les"] == 11:
        flops += 18432
    return {"bytes": steps * arrays * word * n + 32 * n, "flops": steps * flops * n}


def tolerance(case):
    """About four times the distance between `run` and `exact` (the pressure's, which
    starts from zero: 1e-11 in FP64, 1e-3 with FP32 fields; the learned closure's
    BF16 operands move it by 8e-5, the network's own gradient by 2e-3)."""
    if case["kind"] == "train":
        return {"rel": 8e-3}
    if case["precision"] == "mixed":
        return {"rel": 4e-3}
    if case["les"] == 11:
        return {"rel": 4e-4}
    return {"rel": 5e-11}


# ---------------------------------------------------------------------------
# the same in 64 bits with torch
# ---------------------------------------------------------------------------
def _exact_train(case, seed):
    X, T = (t.double() for t in _batch(case, seed))
    p = torch.tensor(_closure(seed)[0], device="cuda").double().requires_grad_(True)
    y = _network(p, X)
    loss = ((y - T) ** 2).sum()
    (loss / y.numel()).backward()
    g = p.grad
    m, v = 0.1 * g, 0.001 * g * g
    new = p.detach() - 1e-3 * (m / 0.1) / (torch.sqrt(v / 0.001) + 1e-8)
    # Adam's first step is the sign of the gradient, which has no value where the gradient is rounding
    return {"loss": loss.detach().reshape(1), "grad": g, "params": new}


def _network(p, x):
    o = 0
    for k, (i, n) in enumerate(((10, 64), (64, 64), (64, 64), (64, 6))):
        x = x @ p[o:o + n * i].reshape(n, i).T + p[o + n * i:o + n * i + n]
        o += n * i + n
        if k < 3:
            x = 0.5 * x * (1 + torch.tanh(math.sqrt(2 / PI) * (x + 0.044715 * x ** 3)))
    return x


class _Exact:
    """One case's solver in 64 bits; fields are (nz, ny, nx), rows j = 0..ny-1."""

    def __init__(self, c, yp):
        self.c, ny = c, c["ny"]
        self.o4, self.per, self.kind = c["kind"] == "o4", c["kind"] == "tg", c["kind"]
        lx, ly, lz = (2 * PI, 2 * PI, 2 * PI) if self.per else ((4 * PI, 2.0, 4 * PI / 3) if c["kind"] in ("o4", "fimp") else (2 * PI, 2.0, PI))
        self.yly = ly
        self.rdx, self.rdz = c["nx"] / lx, c["nz"] / lz
        self.nu = 6.25e-4 if self.per else 2.0 / c["re"]
        yc = 0.5 * (yp[1:] + yp[:-1])
        dyp = np.diff(yp)
        dyc = np.concatenate([[dyp[0]], np.diff(yc), [dyp[-1]]])      # faces 1..ny+1
        dypm = np.concatenate([[dyp[0]], dyp])                         # rows 0..ny
        wy = np.concatenate([dyp, [dyp[-1]]]) / (np.concatenate([dyp, [dyp[-1]]]) + dypm)
        am, ap = 1 / dyp / dyc[:-1], 1 / dyp / dyc[1:]
        amP, apP = am.copy(), ap.copy()
        if not self.per:
            amP[0] = apP[-1] = 0.0
            am[0], ap[0] = 4 / dyc[0] / (dyc[0] + 2 * dyc[1]), 4 / dyc[1] / (dyc[0] + 2 * dyc[1])
            am[-1], ap[-1] = 4 / dyc[-2] / (dyc[-1] + 2 * dyc[-2]), 4 / dyc[-1] / (dyc[-1] + 2 * dyc[-2])
        self.cn = [am.copy(), ap.copy()]                               # Crank-Nicolson rows of ux, uz
        if not self.per:
            self.cn[0][0] *= 2
            self.cn[1][-1] *= 2
        self.cnv = [1 / dyc[:-1] / dypm[:-1], 1 / dyc[:-1] / dyp]      # and of uy
        row = lambda a: torch.tensor(a, device="cuda")[None, :, None]  # noqa: E731
        self.dyp, self.rdyp, self.rdyc, self.rdycp = row(dyp), row(1 / dyp), row(1 / dyc[:-1]), row(1 / dyc[1:])
        self.w1, self.w3 = row(wy[:-1]), row(wy[1:])
        self.am, self.ap, self.vm, self.vp, self.amP, self.apP = (row(a) for a in (am, ap, *self.cnv, amP, apP))
        az = 2 * PI * torch.arange(c["nz"], device="cuda", dtype=torch.float64) / c["nz"]
        ax = 2 * PI * torch.arange(c["nx"] // 2 + 1, device="cuda", dtype=torch.float64) / c["nx"]
        if self.o4:
            wave = lambda a, r: r * r / 288 * (torch.cos(3 * a) - 54 * torch.cos(2 * a) + 783 * torch.cos(a) - 730)  # noqa: E731
        else:
            wave = lambda a, r: 2 * r * r * (torch.cos(a) - 1)  # noqa: E731
        self.lam = wave(az, self.rdz)[:, None] + wave(ax, self.rdx)[None, :]
        if c["kind"] == "les":
            self.delta = row((dyp * lx / c["nx"] * lz / c["nz"]) ** (1 / 3))
            self.dwall = row(np.minimum(yc - yp[0], yp[-1] - yc))

    # neighbours
    @staticmethod
    def X(a, s):
        return torch.roll(a, -s, 2)

    @staticmethod
    def Z(a, s):
        return torch.roll(a, -s, 0)

    def Y(self, a, s, comp):
        """Row j + s (s = -1, 1) with the wall ghosts (no-slip walls at rest) or the periodic rows."""
        if self.per:
            return torch.roll(a, -s, 1)
        if s < 0:
            first = {0: -a[:, :1], 1: torch.zeros_like(a[:, :1]) if self.o4 else -a[:, 1:2], 3: a[:, :1]}[comp]
            return torch.cat([first, a[:, :-1]], 1)
        last = {0: -a[:, -1:], 1: torch.zeros_like(a[:, -1:]), 3: a[:, -1:]}[comp]
        return torch.cat([a[:, 1:], last], 1)

    def div(self, u, v, w):
        dv = (self.Y(v, 1, 1) - v) * self.rdyp
        return self.dst(u, self.X, self.rdx) + dv + self.dst(w, self.Z, self.rdz)

    def dst(self, a, S, r):
        """Staggered difference from the faces to the cell centre."""
        if self.o4:
            return r * ((S(a, -1) - S(a, 2)) / 24 + 1.125 * (S(a, 1) - a))
        return (S(a, 1) - a) * r

    def dback(self, a, S, r):
        """Staggered difference from the cell centres to the face."""
        if self.o4:
            return r * ((S(a, -2) - S(a, 1)) / 24 + 1.125 * (a - S(a, -1)))
        return (a - S(a, -1)) * r

    def poisson(self, src):
        nz, ny, nx = src.shape
        f = torch.fft.fftn(torch.fft.rfft(src, dim=2), dim=(0,))
        if self.per:
            f = torch.fft.fft(f, dim=1)
            mu = 2 * (ny / self.yly) ** 2 * (torch.cos(2 * PI * torch.arange(ny, device="cuda", dtype=torch.float64) / ny) - 1)
            den = self.lam[:, None, :] + mu[None, :, None]
            den[0, 0, 0] = 1.0
            f[0, 0, 0] = 0.0
            f = torch.fft.ifft(f / den, dim=1)
            f[0, :, 0] = f[0, :, 0] - f[0, 0, 0].clone()
        else:
            am, ap = self.amP.flatten(), self.apP.flatten()
            b = torch.empty_like(f.real)
            cp = torch.zeros_like(self.lam)
            for j in range(ny):
                d = -(am[j] + ap[j]) + self.lam - (am[j] * cp if j else 0.0)
                up = ap[j].expand_as(d).clone()
                if j == 0:
                    d[0, 0], up[0, 0], f[0, 0, 0] = 1.0, 0.0, 0.0
                f[:, j] = (f[:, j] - (am[j] * f[:, j - 1] if j else 0.0)) / d
                cp = up / d
                b[:, j] = cp
            for j in range(ny - 2, -1, -1):
                f[:, j] -= b[:, j] * f[:, j + 1]
        return torch.fft.irfft(torch.fft.ifft(f, dim=0), n=nx, dim=2)

    def project(self, u, v, w, alpha):
        """u - alpha grad phi with div = 0, and phi."""
        phi = self.poisson(self.div(u, v, w) / alpha)
        u = u - alpha * self.dback(phi, self.X, self.rdx)
        v = v - alpha * (phi - self.Y(phi, -1, 3)) * self.rdyc
        w = w - alpha * self.dback(phi, self.Z, self.rdz)
        return u, v, w, phi

    def sweep_y(self, r, beta, comp):
        lo, hi = self.cnv if comp == 1 else self.cn
        A = np.diag(1 + beta * (lo + hi)) - beta * np.diag(hi[:-1], 1) - beta * np.diag(lo[1:], -1)
        if comp == 1:
            A[0] = 0.0
            A[0, 0] = 1.0
            r = torch.cat([torch.zeros_like(r[:, :1]), r[:, 1:]], 1)
        return torch.matmul(torch.tensor(np.linalg.inv(A), device="cuda"), r)

    def sweep_periodic(self, r, beta, dim, rd):
        n = r.shape[dim]
        shape = [1, 1, 1]
        shape[dim] = n // 2 + 1
        mu = 1 - 2 * beta * rd * rd * (torch.cos(2 * PI * torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64) / n) - 1)
        return torch.fft.irfft(torch.fft.rfft(r, dim=dim) / mu.reshape(shape), n=n, dim=dim)

    def convect2(self, u, v, w):
        """Convective terms of the 2nd order on the staggered mesh (interpolated y weights)."""
        X, Y, Z, rx, rz = self.X, self.Y, self.Z, self.rdx, self.rdz
        les = self.kind == "les"   # the LES right-hand sides average in y without weights
        w1, w3 = (0.5, 0.5) if les else (self.w1, self.w3)
        mx, mz = (lambda a: a + X(a, -1)), (lambda a: a + Z(a, -1))
        uj = lambda a: w1 * Y(a, -1, 0) + (1 - w1) * a  # noqa: E731  at the lower face
        uJ = lambda a: w3 * a + (1 - w3) * Y(a, 1, 0)   # noqa: E731  at the upper face
        vp = Y(v, 1, 1)
        d = lambda f, S, r: (S(f, 1) - f) * r  # noqa: E731
        h1 = ((X(u, 1) + u) ** 2 - (u + X(u, -1)) ** 2) * rx / 4
        h1 = h1 + (mx(vp) * uJ(u) - mx(v) * uj(u)) * self.rdyp / 2 + d(mx(w) * mz(u), Z, rz) / 4
        h2 = d(uj(u) * mx(v), X, rx) / 2 + ((vp + v) ** 2 - (v + Y(v, -1, 1)) ** 2) * self.rdyc / 4 + d(uj(w) * mz(v), Z, rz) / 2
        h3 = d(mz(u) * mx(w), X, rx) / 4 + (mz(vp) * uJ(w) - mz(v) * uj(w)) * self.rdyp / 2
        h3 = h3 + ((Z(w, 1) + w) ** 2 - (w + Z(w, -1)) ** 2) * rz / 4
        return h1, h2, h3

    def convect4(self, u, v, w):
        X, Y, Z, rx, rz = self.X, self.Y, self.Z, self.rdx, self.rdz
        iu = lambda a, S: (-S(a, -1) + 9 * a + 9 * S(a, 1) - S(a, 2)) / 16  # noqa: E731  face to centre
        ic = lambda a, S: (-S(a, -2) + 9 * S(a, -1) + 9 * a - S(a, 1)) / 16  # noqa: E731  centre to face
        uj = lambda a: self.w1 * Y(a, -1, 0) + (1 - self.w1) * a  # noqa: E731
        uJ = lambda a: self.w3 * a + (1 - self.w3) * Y(a, 1, 0)   # noqa: E731
        up = lambda a: torch.cat([a[:, 1:], torch.zeros_like(a[:, :1])], 1)  # noqa: E731
        vx, vz = ic(v, X), ic(v, Z)
        h1 = self.dback(iu(u, X) ** 2, X, rx) + (up(vx) * uJ(u) - vx * uj(u)) * self.rdyp + self.dst(ic(u, Z) * ic(w, X), Z, rz)
        vp = Y(v, 1, 1)
        h2 = self.dst(vx * uj(u), X, rx) + ((vp + v) ** 2 - (v + Y(v, -1, 1)) ** 2) * self.rdyc / 4 + self.dst(vz * uj(w), Z, rz)
        h3 = self.dst(ic(w, X) * ic(u, Z), X, rx) + (up(vz) * uJ(w) - vz * uj(w)) * self.rdyp + self.dback(iu(w, Z) ** 2, Z, rz)
        return h1, h2, h3

    def lap(self, a, S, r):
        if self.o4:
            return r * r * (-(S(a, -2) + S(a, 2)) / 12 + 4 / 3 * (S(a, -1) + S(a, 1)) - 2.5 * a)
        return r * r * (S(a, 1) - 2 * a + S(a, -1))

    def lapy(self, a, comp):
        lo, hi = (self.vm, self.vp) if comp == 1 else (self.am, self.ap)
        return hi * self.Y(a, 1, comp) - (lo + hi) * a + lo * self.Y(a, -1, comp)

    # subgrid models
    def gradients(self, u, v, w):
        X, Y, Z, rx, rz = self.X, self.Y, self.Z, self.rdx, self.rdz
        vp = Y(v, 1, 1)
        cy = lambda a: ((Y(a, 1, 0) - a) * self.rdycp + (a - Y(a, -1, 0)) * self.rdyc) / 2  # noqa: E731
        c2 = lambda a, S, r: (S(a, 1) - S(a, -1)) * r / 2  # noqa: E731
        um, vm, wm = (X(u, 1) + u) / 2, (vp + v) / 2, (Z(w, 1) + w) / 2
        return [(X(u, 1) - u) * rx, cy(um), c2(um, Z, rz), c2(vm, X, rx), (vp - v) * self.rdyp, c2(vm, Z, rz),
                c2(wm, X, rx), cy(wm), (Z(w, 1) - w) * rz]

    def subgrid(self, u, v, w):
        """Total viscosity and explicit force of the step."""
        d = 0.5 * self.dyp.flatten()  # distance of the first and last centre from its wall
        ut = torch.sqrt(self.nu * 0.5 * (u[:, 0].mean().abs() / d[0] + u[:, -1].mean().abs() / d[-1]))
        G = self.gradients(u, v, w)
        S = [G[0], (G[1] + G[3]) / 2, (G[2] + G[6]) / 2, G[4], (G[5] + G[7]) / 2, G[8]]
        mag = torch.sqrt(2 * (S[0] ** 2 + S[3] ** 2 + S[5] ** 2 + 2 * (S[1] ** 2 + S[2] ** 2 + S[4] ** 2)))
        ypl = self.dwall * ut / self.nu
        nt = (0.1 * (1 - torch.exp(-ypl / 26)) * self.delta) ** 2 * mag
        if self.c["les"] == 10:
            return nt + self.nu, None
        p, n = (torch.tensor(a, device="cuda").double() for a in _closure(self.seed))
        x = torch.stack([g * self.nu / ut ** 2 for g in G] + [ypl.expand_as(G[0])], -1)
        x = (x - n[0:10]) / n[10:20]
        inside = ((x >= n[20:30]) & (x <= n[30:40])).all(-1)
        y = _network(p, x) * n[46:52] + n[40:46]
        t = [torch.where(inside, y[..., q] * ut ** 2, -2 * nt * S[q]) for q in range(6)]
        X, Z, rx, rz = self.X, self.Z, self.rdx, self.rdz
        zero = torch.zeros_like(u[:, :1])
        lowf = lambda a: torch.cat([zero, (a[:, 1:] + a[:, :-1]) / 2], 1)  # noqa: E731  at the lower faces, zero on the walls
        dy = lambda a: (torch.cat([a[:, 1:], zero], 1) - a) * self.rdyp  # noqa: E731
        e = lambda a, S_: (a + S_(a, -1)) / 2  # noqa: E731
        txy, tyz, txz = lowf(e(t[1], X)), lowf(e(t[4], Z)), e(e(t[2], X), Z)
        f1 = (t[0] - X(t[0], -1)) * rx + dy(txy) + (Z(txz, 1) - txz) * rz
        f2 = (X(txy, 1) - txy) * rx + (t[3] - torch.cat([zero, t[3][:, :-1]], 1)) * self.rdyc + (Z(tyz, 1) - tyz) * rz
        f2[:, 0] = 0.0
        f3 = (X(txz, 1) - txz) * rx + dy(tyz) + (t[5] - Z(t[5], -1)) * rz
        return torch.full_like(u, self.nu), (-f1, -f2, -f3)

    def viscous_les(self, u, v, w, nut):
        """Explicit part, y terms for Crank-Nicolson, and the face viscosities of the y solves."""
        X, Y, Z, rx, rz = self.X, self.Y, self.Z, self.rdx, self.rdz
        N = lambda s: torch.cat([2 * self.nu - nut[:, :1], nut[:, :-1]], 1) if s < 0 else torch.cat([nut[:, 1:], 2 * self.nu - nut[:, -1:]], 1)  # noqa: E731
        nm, npl = N(-1), N(1)
        mx, mz = (lambda a: a + X(a, -1)), (lambda a: a + Z(a, -1))
        xl, xu = mx(nut + nm) / 4, mx(nut + npl) / 4            # xy edges below and above
        zl, zu = mz(nut + nm) / 4, mz(nut + npl) / 4            # yz edges
        xz = mx(mz(nut)) / 4                                    # xz edge
        bx, bz = (lambda a: (a - X(a, -1)) * rx), (lambda a: (a - Z(a, -1)) * rz)
        vp = Y(v, 1, 1)
        by = lambda a: (a - Y(a, -1, 0)) * self.rdyc  # noqa: E731
        s11 = (nut * (X(u, 1) - u) - X(nut, -1) * (u - X(u, -1))) * rx * rx
        s33 = (nut * (Z(w, 1) - w) - Z(nut, -1) * (w - Z(w, -1))) * rz * rz
        s22 = self.vp * nut * (vp - v) - self.vm * nm * (v - Y(v, -1, 1))
        dz = lambda f: (Z(f, 1) - f) * rz  # noqa: E731
        dx = lambda f: (X(f, 1) - f) * rx  # noqa: E731
        y1 = self.ap * xu * (Y(u, 1, 0) - u) - self.am * xl * (u - Y(u, -1, 0))
        y3 = self.ap * zu * (Y(w, 1, 0) - w) - self.am * zl * (w - Y(w, -1, 0))
        e1 = 2 * s11 + (xu * bx(vp) - xl * bx(v)) * self.rdyp + dz(xz * (bx(w) + bz(u)))
        e2 = s22 + dx(xl * (by(u) + bx(v))) + dz(zl * (by(w) + bz(v)))
        e3 = 2 * s33 + dx(xz * (bz(u) + bx(w))) + (zu * bz(vp) - zl * bz(v)) * self.rdyp
        return (e1, e2, e3), (y1, s22, y3), ((xl, xu), (nm, nut), (zl, zu))

    def sweep_les(self, r, betaT, vis, comp):
        lo, hi = self.cnv if comp == 1 else self.cn
        ny = r.shape[1]
        r = r.clone()
        cp = torch.zeros_like(r)
        for j in range(ny):
            a, cc = -betaT * vis[0][:, j] * lo[j], -betaT * vis[1][:, j] * hi[j]
            b = 1 - a - cc
            if comp == 1 and j == 0:
                a, b, cc, r[:, 0] = a * 0, b * 0 + 1, cc * 0, 0.0
            m = b - a * cp[:, j - 1] if j else b
            r[:, j] = (r[:, j] - (a * r[:, j - 1] if j else 0.0)) / m
            cp[:, j] = cc / m
        for j in range(ny - 2, -1, -1):
            r[:, j] -= cp[:, j] * r[:, j + 1]
        return r

    def step(self, q, p):
        c, nu, dt = self.c, self.nu, self.c["dt"]
        X, Y, Z, rx, rz = self.X, self.Y, self.Z, self.rdx, self.rdz
        u, v, w = q
        nut, force = self.subgrid(u, v, w) if self.kind == "les" else (None, None)
        hist = None
        for gam, the in ((8 / 15, 0.0), (5 / 12, -17 / 60), (3 / 4, -5 / 12)):
            alp = gam + the
            gam, the, alpha, beta = gam * dt, the * dt, alp * dt, 0.5 * alp * nu * dt
            h = self.convect4(u, v, w) if self.o4 else self.convect2(u, v, w)
            lx = [self.lap(a, X, rx) for a in (u, v, w)]
            lz = [self.lap(a, Z, rz) for a in (u, v, w)]
            ly = [self.lapy(a, k) for a, k in ((u, 0), (v, 1), (w, 0))]
            if self.kind == "fimp":
                conv, visc = [-a for a in h], [2 * beta * (a + b + d) for a, b, d in zip(lx, ly, lz)]
            elif self.per:
                conv, visc = [-a + nu * (b + d + e) for a, b, d, e in zip(h, lx, ly, lz)], [0.0] * 3
            elif self.kind == "les":
                ex, ycn, vis = self.viscous_les(u, v, w, nut)
                conv = [-a + b + (force[k] if force else 0.0) for k, (a, b) in enumerate(zip(h, ex))]
                visc = [alp * dt * a for a in ycn]
            else:
                conv, visc = [-a + nu * (b + d) for a, b, d in zip(h, lx, lz)], [2 * beta * a for a in ly]
            grad = [self.dback(p, X, rx), (p - Y(p, -1, 3)) * self.rdyc, self.dback(p, Z, rz)]
            r = [gam * a - alpha * b + d + (the * e if the else 0.0) for a, b, d, e in zip(conv, grad, visc, hist or conv)]
            hist = conv
            per_area = 1.0 / (c["nx"] * c["nz"]) / self.yly
            if self.o4:
                r[0] = r[0] - alpha * nu * ((lx[0] + ly[0] + lz[0]) * self.dyp).sum() * per_area
            elif not self.per:
                r[0] = r[0] + alp * (1.0 - (u * self.dyp).sum() * per_area)
            if self.kind == "fimp":
                r = [self.sweep_periodic(self.sweep_periodic(a, beta, 2, rx), beta, 0, rz) for a in r]
            if self.kind == "les":
                r = [self.sweep_les(a, 0.5 * alp * dt, vis[k], k) for k, a in enumerate(r)]
            elif not self.per:
                r = [self.sweep_y(a, beta, k) for k, a in enumerate(r)]
            u, v, w = u + r[0], v + r[1], w + r[2]
            if self.kind == "fimp":
                p = p - 0.5 * nu * self.div(u, v, w)
            u, v, w, phi = self.project(u, v, w, alpha)
            if self.kind in ("fimp", "tg"):
                p = p + phi
            elif self.kind == "les":
                bT = 0.5 * alp * dt
                nm = torch.cat([2 * nu - nut[:, :1], nut[:, :-1]], 1)
                npl = torch.cat([nut[:, 1:], 2 * nu - nut[:, -1:]], 1)
                p = p + phi - bT * (self.rdyp * self.rdycp * (npl + nut) / 2 * (Y(phi, 1, 3) - phi) -
                                    self.rdyp * self.rdyc * (nut + nm) / 2 * (phi - Y(phi, -1, 3)))
            else:
                p = p + phi - beta * (self.apP * (Y(phi, 1, 3) - phi) - self.amP * (phi - Y(phi, -1, 3)))
        return (u, v, w), p


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    yp = _mesh(case)
    e = _Exact(case, yp)
    e.seed = seed
    u, v, w, p = _start(case, yp, seed)
    q = e.project(u, v, w, 1.0)[:3]
    for _ in range(case["nsteps"] // case["calls"] * case["calls"]):
        q, p = e.step(q, p)
    r = {"stat": None} if case["kind"] == "o4" else {}
    r.update(zip(NAMES, (*q, p)))
    return r
