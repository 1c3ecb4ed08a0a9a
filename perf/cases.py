"""What the framework's speed is measured on: calls that its users make, over the sizes that they make them at.

A simulation is a `Solver` that a program creates once and steps; one pass advances it by the steps that lie between two
looks at its fields and reads the fields back into page-locked host arrays.  The warm start's network trains on one
volume per pass or corrects one volume.  Sizes are those of `littleharsh_gb300.workloads`, or lie between them.

Fields are a laminar profile between the canopy tips plus a random perturbation with energy in every mode, falling off as
in a turbulent channel and smooth in y, projected divergence free by the solver as a program does before its first step.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import littleharsh_gb300 as lh
from littleharsh_gb300 import srnet, workloads

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _sim(name, base, **kw):
    """A simulation case: kind, steps per pass and the quantities of `Config` that differ between workloads."""
    keys = ("Re", "ngalx", "ngalz", "ny", "posth", "dsty", "dstx", "dstz", "ntilex", "ntilez", "flag_ctpress")
    c = {"name": name, "kind": "step", "steps": 1, "precision": "fp64", "ngalx2": 0, "ngalz2": 0}
    c.update({k: base[k] for k in keys})
    c.update(kw)
    return c


def listed():
    w = workloads
    mid = dict(w.MID288)
    return [
        # the smallest simulation: the coarse grid of the warm start, where launches and latency count
        _sim("coarse48_fp64", w.CONFIG1_COARSE, steps=4),
        # the Re_tau 180 channel, the everyday run, in both precisions
        _sim("channel96_fp64", w.CONFIG1, steps=4),
        _sim("channel96_mixed", w.CONFIG1, steps=4, precision="mixed"),
        # the same run's output interval: a few steps, then plane, conditional and spectral statistics and a new time
        # step from the CFL number, as the C driver's main loop does
        _sim("interval96_fp64", w.CONFIG1, kind="interval", steps=2),
        # odd numbers throughout: unlike x and z, transform lengths with many threes, driven by a pressure gradient
        _sim("ragged162x108_fp64", w.CONFIG1, ngalx=162, ngalz=108, ny=101, dsty=11, dstx=3, dstz=5, ntilex=9, ntilez=6,
             flag_ctpress=1, steps=2),
        # a mid-size run, and the same with the reference's variable-resolution bands (a coarser channel core)
        _sim("mid288_fp64", mid),
        _sim("bands288_192_fp64", mid, ngalx2=192, ngalz2=192),
        # four replicas of two sizes advanced together, a cut of the 16-replica ensemble
        _sim("ensemble4_fp64", w.CONFIG1, kind="ensemble", ngalx=144, ngalz=144, ny=129, dsty=12, dstx=3, dstz=6,
             members=4, step_up=4, mode="streams"),
        # the Re_tau 550 production run, in both precisions
        _sim("production576_fp64", w.CONFIG2),
        _sim("production576_mixed", w.CONFIG2, precision="mixed"),
        # the warm start's network: one training step on the Re_tau 180 volume, and the correction of its 2x grid
        {"name": "train96", "kind": "train", "Y": 130, "Z": 96, "X": 96},
        {"name": "infer192", "kind": "infer", "Y": 258, "Z": 192, "X": 192},
    ]


# transform lengths (2, 3 and 4 only, even, a multiple of 3) from the coarse grid's to the production run's
_LENGTHS = [48, 54, 72, 96, 108, 144, 162, 192, 216, 288, 324, 384, 432, 486, 576]


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["interval", "ensemble", "train", "infer"])
    if kind == "train":
        return {"kind": kind, "Y": rng.randint(48, 130), "Z": rng.choice([48, 64, 80, 96]), "X": rng.choice([32, 64, 96])}
    if kind == "infer":
        return {"kind": kind, "Y": rng.randint(48, 258), "Z": rng.choice([48, 96, 144, 192]),
                "X": rng.choice([64, 96, 128, 192])}
    small = [n for n in _LENGTHS if n <= 288]
    ngx = rng.choice(small if kind != "step" else _LENGTHS)
    ngz = rng.choice([n for n in _LENGTHS if ngx / 2 <= n <= 2 * ngx and (kind == "step" or n <= 288)])
    # y points grow with the plane, odd as input.in has them
    ny = int(round(0.75 * math.sqrt(ngx * ngz) * math.exp(rng.uniform(-0.25, 0.12)))) // 2 * 2 + 17
    tx = rng.choice([t for t in (4, 6, 8, 9, 12, 16, 18, 24) if ngx % t == 0 and ngx // t >= 4])
    tz = rng.choice([t for t in (3, 4, 6, 8, 9, 12) if ngz % t == 0 and ngx % t == 0 and ngz // t >= 4])
    posth = rng.choice([0.1, 0.2])
    c = _sim("", workloads.CONFIG1, kind=kind, Re=rng.choice([2800.0, 4500.0, 6900.0, 10000.0]), ngalx=ngx, ngalz=ngz,
             ny=ny, posth=posth, dsty=max(3, int(ny * posth * rng.uniform(0.6, 0.9))), ntilex=tx, ntilez=tz,
             dstx=max(1, ngx // tx // 4), dstz=max(1, ngz // tz // 4), flag_ctpress=rng.choice([0, 0, 1]),
             steps=max(1, min(4, 200 // ngx)))
    del c["name"]
    if kind == "step":
        c["precision"] = rng.choice(["fp64", "fp64", "mixed"])
        if rng.random() < 0.2 and ngx >= 96 and ngz >= 96:
            c["ngalx2"] = rng.choice([n for n in _LENGTHS if ngx / 2 <= n < ngx])
            c["ngalz2"] = rng.choice([n for n in _LENGTHS if ngz / 2 <= n < ngz])
    if kind == "ensemble":
        c.update(members=rng.randint(2, 4), step_up=rng.choice([0, 4, 8]), mode=rng.choice(["streams", "batched"]),
                 steps=1)
    return c


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------

def _config(c, member=0):
    kw = {k: c[k] for k in ("Re", "ngalx", "ngalz", "ny", "posth", "dsty", "dstx", "dstz", "ntilex", "ntilez",
                            "flag_ctpress", "ngalx2", "ngalz2")}
    if member % 2:  # every other replica has more y points
        kw["ny"] += c["step_up"]
    return lh.Config(alp=1.0, bet=2.0, dyq=13.6, ppp=5, geometry_type=3, mpgx=-0.004 if c["flag_ctpress"] else 0.0,
                     CFL=0.3, **kw)


def _fields(g, prm, seed, banded):
    """u1, u2, u3, p (complex128, [level][kz][kx]) on DEV for grid arrays `g` and parameters `prm`."""
    ngx, ngz = prm.Ngal[4], prm.Ngal[5]
    nkx, nz = ngx // 3 + 1, 2 * (ngz // 3)
    nyu = g["yu"].size
    gen = torch.Generator().manual_seed(int(seed))
    kx = torch.arange(nkx, dtype=torch.float64)[None, :] * prm.alp
    kz = torch.fft.fftfreq(nz, 1.0 / nz, dtype=torch.float64)[:, None] * prm.bet
    k2 = kx * kx + kz * kz
    amp = (1.0 + k2 / 36.0) ** (-4.0 / 3.0) * torch.exp(-2.0 * (k2 / float(k2.max())))
    amp[nz // 2, :] = 0.0  # the lone -nz/2 mode
    amp[0, 0] = 0.0
    if banded:  # modes of the middle band only: the others may not cross it
        amp[:, (prm.Ngal[8] // 3 + 1):] = 0.0
        h2 = prm.Ngal[9] // 3
        amp[h2:nz - h2 + 1, :] = 0.0
    modes, out = 6, []
    for name, scale in (("yu", 0.12), ("yv", 0.08), ("yu", 0.10), ("yu", 0.02)):
        y = torch.from_numpy(np.ascontiguousarray(g[name]))
        if len(out) == 3:
            y = y[1:nyu - 1]  # the pressure's levels
        c = torch.complex(torch.randn(modes, nz, nkx, generator=gen, dtype=torch.float64),
                          torch.randn(modes, nz, nkx, generator=gen, dtype=torch.float64)) * amp
        neg = torch.conj(torch.roll(torch.flip(c[:, :, 0], (1,)), 1, 1))
        c[:, :, 0] = 0.5 * (c[:, :, 0] + neg)  # a real field's kx = 0 line
        w = torch.full((nkx,), 2.0, dtype=torch.float64)
        w[0] = 1.0
        c *= scale / torch.sqrt(((c.abs() ** 2) * w).sum((0, 1, 2)))
        ye = torch.clamp(y.abs() / float(y.abs().max()), max=1.0)
        phi = torch.stack([torch.cos((m + 0.5) * math.pi * (y + 0.3 * m)) for m in range(modes)], 1) * (1 - ye ** 4)[:, None]
        f = torch.tensordot(phi.to(torch.complex128).to(DEV), c.to(DEV), dims=1)
        if len(out) == 0:
            f[:, 0, 0] += torch.where(y.abs() < 1.0, 1.5 * (1.0 - y * y), torch.zeros_like(y)).to(DEV)
        if len(out) == 1:
            f[0] = 0.0
            f[-1] = 0.0
        out.append(f.contiguous())
    return out


def _pinned(shape):
    return torch.empty(shape, dtype=torch.complex128, pin_memory=DEV == "cuda").numpy()


def _time_step(x):
    """A CFL time step as a program would note it down: three digits."""
    return float("%.3g" % x)


def _solver(c, seed, member=0):
    cfg = _config(c, member)
    s = lh.Solver(cfg, precision=lh.PREC_MIXED if c["precision"] == "mixed" else lh.PREC_FP64)
    host = [_pinned(s.shape(x)) for x in "uvup"]
    for h, f in zip(host, _fields(s.grid, s.params, 1000 * int(seed) + member, bool(c["ngalx2"]))):
        torch.from_numpy(h).copy_(f)
    if DEV == "cuda":
        torch.cuda.synchronize()
    s.set_fields(*host)
    s.set_time(0.0, 1.0, cfg.mpgx)
    s.project()
    s.set_time(0.0, _time_step(s.cfl_dt(cfg.CFL)), cfg.mpgx)
    return s, host


def _net_input(Y, Z, X, seed):
    """bf16 network input, the lifted base and the target of the Re_tau 180 geometry's proportions."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.zeros(Y, Z, X, srnet.CIN0, dtype=torch.float32, device=DEV)
    y = torch.linspace(-1.2, 1.2, Y, device=DEV)[:, None, None]
    x[..., :3] = 0.3 * torch.randn(Y, Z, X, 3, generator=g, device=DEV)
    x[..., 0:1] += (1.5 * (1.0 - y * y).clamp(min=0.0))[..., None]
    px = torch.arange(X, device=DEV) % 8 < 2
    pz = torch.arange(Z, device=DEV) % 16 < 4
    x[..., 3] = ((y.abs() > 1.0) & (pz[None, :, None] & px[None, None, :])).float()
    x[..., 4] = y
    base = x[..., :3].reshape(-1, 3).contiguous()
    target = base + 0.1 * torch.randn(base.shape, generator=g, device=DEV)
    return x.to(torch.bfloat16), base, target


def _net_params(seed):
    """Weights of a network in training: the initial ones with the last layers moved off zero."""
    params = srnet.init_params(int(seed) % 1000003)
    rng = np.random.default_rng(int(seed))
    w, b = params[-1]
    w[:, :3] = (rng.standard_normal((27, 3, w.shape[2])) * 0.02).astype(np.float32)
    return [(w, (0.01 * rng.standard_normal(b.shape)).astype(np.float32) if i < len(params) - 1 else b)
            for i, (w, b) in enumerate(params)]


def prepare(case, seed):
    c = case
    if c["kind"] in ("train", "infer"):
        net = srnet.SRNet(params=_net_params(seed), lr=1e-4)
        x, base, target = _net_input(c["Y"], c["Z"], c["X"], seed)
        return {"kind": c["kind"], "net": net, "x": x, "base": base, "target": target,
                "loss": torch.zeros(1, dtype=torch.float64, device=DEV)}
    if c["kind"] == "ensemble":
        made = [_solver(c, seed, m) for m in range(c["members"])]
        ens = lh.Ensemble([s for s, _ in made], mode=lh.ENS_BATCHED if c["mode"] == "batched" else lh.ENS_STREAMS)
        return {"kind": "ensemble", "steps": c["steps"], "ens": ens, "made": made}
    s, host = _solver(c, seed)
    return {"kind": c["kind"], "steps": c["steps"], "s": s, "host": host}


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "step":
        s = state["s"]
        s.step(state["steps"])
        return s.get_fields(out=state["host"])
    if kind == "interval":
        s = state["s"]
        s.step(state["steps"])
        s.stats_accumulate()
        s.cond_accumulate()
        s.spectra_accumulate()
        now = s.time()
        s.set_time(now["t"], s.cfl_dt(s.config.CFL), now["mpgx"])
        spectra = s.spectra_flush()[1]
        return {"fields": s.get_fields(out=state["host"]), "mpgx": now["mpgx"], "Qx": now["Qx"], "dt": s.time()["dt"],
                "stats": s.stats_flush()[1], "cond": s.cond_flush()[1], "spectra": spectra}
    if kind == "ensemble":
        state["ens"].step(state["steps"])
        return [s.get_fields(out=host) for s, host in state["made"]]
    net = state["net"]
    if kind == "infer":
        return net.forward(state["x"])
    net.zero_grad()
    state["loss"].zero_()
    corr = net.forward(state["x"], keep=True)
    net.backward(net.loss_grad(corr, state["base"], state["target"], state["loss"]))
    net.adam_step()
    return {"corr": corr, "loss": state["loss"], "grad": net.grad, "master": net.master}


# ---------------------------------------------------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------

def _sim_work(c, member=0):
    nkx, nz = c["ngalx"] // 3 + 1, 2 * (c["ngalz"] // 3)
    nyu = c["ny"] + (c.get("step_up", 0) if member % 2 else 0) + 2 * c["dsty"] + 1
    spec = nkx * nz * nyu * 16.0  # one field's bytes
    # a band of coarser planes in the middle: about three quarters of the levels
    share = 1.0 if not c["ngalx2"] else 0.25 + 0.75 * c["ngalx2"] * c["ngalz2"] / (c["ngalx"] * c["ngalz"])
    pts = c["ngalx"] * c["ngalz"] * nyu * share
    # per substage: u, w, v, p and the last nonlinear term read, u, w, v, p and the new term written
    state = 3 * c["steps"] * 14 * spec
    # nine real transforms of each plane (three fields there, six products back) at 5/2 n log2 n, twelve flops a point
    # for products and interpolation, and four tridiagonal solves of complex columns
    flops = 3 * c["steps"] * (9 * 2.5 * pts * math.log2(c["ngalx"] * c["ngalz"]) + 12 * pts + 120 * nkx * nz * nyu)
    out = 4 * spec
    if c["kind"] == "interval":
        out += 4 * spec + 2.5 * spec  # the statistics read the fields once and return five real spectra
        flops += 40 * nkx * nz * nyu
    return state + out, flops


def work(case):
    c = case
    if c["kind"] in ("train", "infer"):
        nvox = float(c["Y"] * c["Z"] * c["X"])
        mac = sum(27.0 * ci * co for ci, co in srnet.layer_shapes())
        if c["kind"] == "infer":
            return {"bytes": nvox * (16 * 2 + 16 * 4), "flops": 2 * mac * nvox}
        acts = sum(co for _, co in srnet.layer_shapes()[:-1])
        return {"bytes": nvox * (16 * 2 + 2 * 2 * acts + 16 * 4 + 2 * 3 * 4), "flops": 6 * mac * nvox}
    if c["kind"] == "ensemble":
        parts = [_sim_work(c, m) for m in range(c["members"])]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    b, f = _sim_work(c)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------------------------------------
# the same results in 64 bits, from torch alone
# ---------------------------------------------------------------------------------------------------------------------

class _Exact:
    """The RK3 step of one resolution in FP64 with torch's transforms and plain loops over y."""

    A = (4.0 / 15.0, 1.0 / 15.0, 1.0 / 6.0)
    G = (8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0)
    C = (0.0, -17.0 / 60.0, -5.0 / 12.0)
    D = (8.0 / 15.0, 2.0 / 15.0, 1.0 / 3.0)

    def __init__(self, c, seed, member=0):
        cfg = _config(c, member)
        prm, g, lu, lv = lh.setup(cfg.to_input())
        self.c, self.cfg, self.prm = c, cfg, prm
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        self.ngx, self.ngz = c["ngalx"], c["ngalz"]
        self.nkx, self.nz = self.ngx // 3 + 1, 2 * (self.ngz // 3)
        self.yu, self.yv = t(g["yu"]), t(g["yv"])
        self.du, self.dv = t(g["dyu2i"]), t(g["dyv2i"])
        self.cu, self.cv = prm.ddthetavi * t(g["dthdyu"]), prm.ddthetavi * t(g["dthdyv"])
        self.nyu, self.nyv, self.j0 = self.yu.numel(), self.yv.numel(), prm.N[3]
        self.kx = (prm.alp * torch.arange(self.nkx, dtype=torch.float64, device=DEV))[None, None, :]
        self.kz = (prm.bet * torch.fft.fftfreq(self.nz, 1.0 / self.nz, dtype=torch.float64, device=DEV))[None, :, None]
        self.k2 = -(self.kx ** 2 + self.kz ** 2)[0]
        self.gw = np.array(prm.gridweighting).reshape(2, 3).T
        self.wc = torch.zeros_like(self.yu)
        self.wc[1:-1] = (self.yu[1:-1] - self.yv[:-1]) / (self.yv[1:] - self.yv[:-1])
        self.wf = (self.yv[1:-1] - self.yu[1:-2]) / (self.yu[2:-1] - self.yu[1:-2])  # faces 1..nyv-2
        self.masks = self._masks(lu, lv)
        self.u, self.v, self.w, self.p = _fields(g, prm, 1000 * int(seed) + member, False)
        self.n = [torch.zeros_like(x) for x in (self.u, self.v, self.w)]
        self.mpgx, self.dt = cfg.mpgx, 1.0
        self.pressure(0, keep_p=True)
        self.QxT = self.flow()
        self.dt = _time_step(self.cfl())

    def _masks(self, lu, lv):
        """Processed planes of the u and v grids: {level: (solid points, whether it is a tip plane)}."""
        N, G, dsty = self.prm.N, self.prm.Ngal, self.prm.dsty
        g4, g3 = G[15], G[14]
        at = lambda row, band: N[4 * band + row - 1]  # noqa: E731
        ur = [(-dsty + 1, 0), (g4 - dsty + 1, g4)]
        vr = [(-dsty, -1), (g3 - dsty + 2, g3 + 1)]
        tips = ((0, g4 - dsty + 1), (-1, g3 - dsty + 2))
        out = []
        for pts, ranges, lo, hi, tip in ((lu, ur, at(4, 0) + 1, at(4, 3), tips[0]), (lv, vr, at(3, 0) + 1, at(3, 3), tips[1])):
            planes = {}
            for a, b in ranges:
                for j in range(max(a, lo), min(b, hi) + 1):
                    planes[j - self.j0] = [np.zeros((self.ngz, self.ngx), bool), j in tip]
            for i, k, j in pts:
                if j - self.j0 in planes:
                    planes[j - self.j0][0][k - 1, i - 1] = True
            out.append({j: (torch.from_numpy(m).to(DEV), tip) for j, (m, tip) in planes.items()})
        return out

    def phys(self, f):
        h = self.nz // 2
        g = torch.zeros(f.shape[0], self.ngz, self.nkx, dtype=f.dtype, device=f.device)
        g[:, :h], g[:, self.ngz - h:] = f[:, :h], f[:, h:]
        g = torch.fft.ifft(g, dim=1, norm="forward")
        g[:, :, 0] = g[:, :, 0].real.to(g.dtype)
        return torch.fft.irfft(g, n=self.ngx, dim=2, norm="forward")

    def spec(self, x):
        h = self.nz // 2
        g = torch.fft.rfft(x, dim=2, norm="forward")[:, :, :self.nkx]
        g = torch.fft.fft(g, dim=1, norm="forward")
        return torch.cat([g[:, :h], g[:, self.ngz - h:]], 1)

    def blocks(self, lo, hi):
        n = max(1, int(2e8 // (self.ngx * self.ngz)))
        return [(a, min(a + n, hi)) for a in range(lo, hi, n)]

    def cfl(self):
        dyc = torch.zeros_like(self.yu)
        dyc[1:-1] = 1.0 / (self.yv[1:] - self.yv[:-1])
        dxi, dzi = self.ngx * self.prm.alp / (2 * math.pi), self.ngz * self.prm.bet / (2 * math.pi)
        most = 0.0
        for a, b in self.blocks(1, self.nyu - 1):
            v = self.phys(self.centre_v(a, b))
            m = self.phys(self.u[a:b]).abs() * dxi + v.abs() * dyc[a:b, None, None] + self.phys(self.w[a:b]).abs() * dzi
            most = max(most, float(m.max()))
        dyw = float(self.yv[1] - self.yv[0])
        dtv = self.prm.Re / (float((self.prm.alp * (self.nkx - 1)) ** 2 + (self.prm.bet * (self.nz // 2 - 1)) ** 2) + 4 / dyw ** 2)
        return self.cfg.CFL * min(1.0 / most, dtv)

    def centre_v(self, a, b):
        """v at the centres a..b-1."""
        lo = self.v[a - 1:b - 1].clone()
        hi = self.v[a:b].clone()
        if a == 1:
            lo[0] = 0.0
        if b == self.nyv:
            hi[-1] = 0.0
        return lo + self.wc[a:b, None, None] * (hi - lo)

    def flow(self):
        nn = self.prm.nn
        q = self.u[1 - self.j0:nn + 2 - self.j0, 0, 0].real
        return float(((self.yv[1 - self.j0:nn + 2 - self.j0] - self.yv[-self.j0:nn + 1 - self.j0]) * q).sum())

    @staticmethod
    def thomas(a, b, c, r):
        """Solve the tridiagonal systems with diagonals a, b, c (levels first; scalars or planes per level) in place of r."""
        n = r.shape[0]
        cp = [None] * n
        inv = 1.0 / b[0]
        cp[0] = c[0] * inv
        r[0] = r[0] * inv
        for j in range(1, n):
            inv = 1.0 / (b[j] - a[j] * cp[j - 1])
            cp[j] = c[j] * inv
            r[j] = (r[j] - a[j] * r[j - 1]) * inv
        for j in range(n - 2, -1, -1):
            r[j] -= cp[j] * r[j + 1]
        return r

    def products(self):
        """The products on centres (uu, uw, ww, vv) and faces (uv, vw), zero on ghost centres and wall faces."""
        cs = [torch.zeros_like(self.u) for _ in range(4)]
        fs = [torch.zeros_like(self.v) for _ in range(2)]
        for a, b in self.blocks(1, self.nyu - 1):
            u, w, v = self.phys(self.u[a:b]), self.phys(self.w[a:b]), self.phys(self.centre_v(a, b))
            for o, x in zip(cs, (u * u, u * w, w * w, v * v)):
                o[a:b] = self.spec(x)
        for a, b in self.blocks(1, self.nyv - 1):
            k = self.wf[a - 1:b - 1, None, None]
            v = self.phys(self.v[a:b])
            for o, f in zip(fs, (self.u, self.w)):
                o[a:b] = self.spec(self.phys(f[a:b] + k * (f[a + 1:b + 1] - f[a:b])) * v)
        return cs + fs

    def lap(self, f, d, k2):
        d = d[:, :, None, None]
        return d[1:-1, 0] * f[:-2] + (k2 + d[1:-1, 1]) * f[1:-1] + d[1:-1, 2] * f[2:]

    def helmholtz(self, d, beta, lo, hi, n):
        a, b, c = (-beta * d[:, 0]).tolist(), (1.0 - beta * d[:, 1]).tolist(), (-beta * d[:, 2]).tolist()
        a[0], b[0], c[0] = 0.0, 1.0, lo
        a[n - 1], b[n - 1], c[n - 1] = hi, 1.0, 0.0
        return a[:n], b[:n], c[:n]

    def substage(self, k):
        dt, Re = self.dt, self.prm.Re
        beta = self.A[k] * dt / Re
        uu, uw, ww, vv, uv, vw = self.products()
        new = [torch.zeros_like(x) for x in self.n]
        ikx, ikz, cu, cv = 1j * self.kx, 1j * self.kz, self.cu[:, None, None], self.cv[:, None, None]
        new[0][1:-1] = ikx * uu[1:-1] + ikz * uw[1:-1] + cu[1:-1] * (uv[1:] - uv[:-1])
        new[2][1:-1] = ikx * uw[1:-1] + ikz * ww[1:-1] + cu[1:-1] * (vw[1:] - vw[:-1])
        new[1][1:-1] = ikx * uv[1:-1] + ikz * vw[1:-1] + cv[1:-1] * (vv[2:-1] - vv[1:-2])
        del uu, uw, ww, vv, uv, vw
        grad = [ikx * self.p, cv[1:-1] * (self.p[1:] - self.p[:-1]), ikz * self.p]
        fields, r = [self.u, self.v, self.w], []
        for q in range(3):
            d = self.dv if q == 1 else self.du
            rhs = torch.zeros_like(fields[q])
            x = self.A[k] / Re * self.lap(fields[q], d, self.k2) - self.C[k] * self.n[q][1:-1] - self.D[k] * grad[q] - self.G[k] * new[q][1:-1]
            if q == 0:
                x[:, 0, 0] -= self.D[k] * self.mpgx
            rhs[1:-1] = (fields[q][1:-1] + dt * x) / (1.0 - beta * self.k2)
            for j, (m, tip) in self.masks[1 if q == 1 else 0].items():
                plane = self.phys(rhs[j:j + 1])
                ly = torch.zeros_like(plane)
                if tip:
                    ly = -beta * self.phys(self.lap(fields[q][j - 1:j + 2], d[j - 1:j + 2], 0.0))
                rhs[j:j + 1] = self.spec(torch.where(m, ly, plane))
            r.append(rhs)
        self.n = new
        n = self.nyu
        gl, gh = float(self.gw[1, 0]), float(self.gw[1, 1])
        self.u = self.thomas(*self.helmholtz(self.du, beta, gl, gh, n), r[0])
        self.w = self.thomas(*self.helmholtz(self.du, beta, gl, gh, n), r[2])
        self.v = self.thomas(*self.helmholtz(self.dv, beta, 0.0, 0.0, self.nyv), r[1])
        if self.prm.flag_ctpress == 0:
            nn, j0 = self.prm.nn, self.j0
            x = torch.full((nn + 3,), -self.D[k] * dt, dtype=torch.float64, device=DEV)
            x[0] = x[-1] = 0.0
            x = self.thomas(*self.helmholtz(self.du[-j0:nn + 3 - j0], beta, gl, gh, nn + 3), x)
            q1 = float(((self.yv[1 - j0:nn + 2 - j0] - self.yv[-j0:nn + 1 - j0]) * x[:nn + 1]).sum())
            g = (self.QxT - self.flow()) / q1
            self.mpgx += g
            self.u[-j0:nn + 3 - j0, 0, 0] += g * x
        self.pressure(k)

    def pressure(self, k, keep_p=False):
        s = 2.0 * self.A[k] * self.dt
        cu, cv = self.cu[:, None, None], self.cv[:, None, None]
        r = (1j * self.kx * self.u[1:-1] + 1j * self.kz * self.w[1:-1] + cu[1:-1] * (self.v[1:] - self.v[:-1])) / s
        n = self.nyu - 2
        up = (self.cu[1:-1] * self.cv[1:]).tolist()    # towards the face above
        down = (self.cu[1:-1] * self.cv[:-1]).tolist()  # towards the face below
        zero = torch.zeros_like(self.k2)
        a = [down[j] + zero for j in range(n)]
        c = [up[j] + zero for j in range(n)]
        b = [self.k2 - (up[j] if j < n - 1 else 0.0) - (down[j] if j > 0 else 0.0) for j in range(n)]
        dy = float(self.yu[2 - self.j0] - self.yu[1 - self.j0])
        b[0] = b[0].clone()
        b[0][0, 0], c[0][0, 0], r[0, 0, 0] = 1.0 / dy ** 2, 0.0, 0.0
        psi = self.thomas(a, b, c, r)
        if not keep_p:
            self.p = self.p + psi
        self.u[1:-1] -= s * 1j * self.kx * psi
        self.w[1:-1] -= s * 1j * self.kz * psi
        self.v[1:-1] -= s * cv[1:-1] * (psi[1:] - psi[:-1])
        self.v[0] = 0.0
        self.v[-1] = 0.0
        for f in (self.u, self.w):
            f[0] = -float(self.gw[0, 0]) * f[1]
            f[-1] = -float(self.gw[2, 1]) * f[-2]

    def step(self, n):
        for _ in range(n):
            for k in range(3):
                self.substage(k)
        return [self.u, self.v, self.w, self.p]

    def statistics(self):
        """Plane and conditional sums and spectra of the present fields, as dicts and lists laid out as the solver's.
        The plane mean of v is zero in a divergence-free field, so its sum is rounding alone."""
        np_ = lambda x: x.cpu().numpy()  # noqa: E731
        u, v, w, p = (self.phys(f) for f in (self.u, self.v, self.w, self.p))
        vc, wf = torch.zeros_like(self.u), torch.zeros_like(self.v)
        vc[1:-1] = self.v[:-1] + self.wc[1:-1, None, None] * (self.v[1:] - self.v[:-1])
        wf[1:-1] = self.w[1:-2] + self.wf[:, None, None] * (self.w[2:-1] - self.w[1:-2])
        om = self.phys(self.cv[:, None, None] * (self.w[1:] - self.w[:-1]) - 1j * self.kz * self.v)
        spectra = [f.abs() ** 2 for f in (self.u, self.v, self.w)] + [(self.u * vc.conj()).real, self.p.abs() ** 2]
        vc, wf = self.phys(vc), self.phys(wf)
        s = lambda x: np_(x.sum((1, 2)))  # noqa: E731
        stats = {"Um": s(u), "U2m": s(u * u), "Vm": None, "V2m": s(v * v), "Wm": s(w), "W2m": s(w * w), "Pm": s(p),
                 "P2m": s(p * p), "UVm": s(u * vc), "UWm": s(u * w), "VWm": s(v * wf), "wxm": s(om), "wx2m": s(om * om)}
        at = lambda row, band: self.prm.N[4 * band + row - 1]  # noqa: E731
        nju, njv, njp = at(4, 1) - at(4, 0) + 1, at(3, 1) - at(3, 0) + 1, at(4, 1) - at(4, 0) - 1
        tz, tx = self.cfg.ntilez, self.cfg.ntilex

        def fold(x, nj, sign=1.0):
            y = x[:nj] + sign * torch.flip(x, (0,))[:nj]
            return np_(y.reshape(nj, tz, self.ngz // tz, tx, self.ngx // tx).sum((1, 3)))

        cond = {"UmC": fold(u, nju), "U2mC": fold(u * u, nju), "WmC": fold(w, nju), "W2mC": fold(w * w, nju),
                "UVmC": fold(u * vc, nju, -1.0), "UWmC": fold(u * w, nju), "VmC": fold(v, njv, -1.0),
                "V2mC": fold(v * v, njv), "VWmC": fold(v * wf, njv, -1.0), "PmC": fold(p, njp), "P2mC": fold(p * p, njp),
                "wxmC": fold(om, njv), "wx2mC": fold(om * om, njv)}
        return stats, cond, [np_(x.reshape(x.shape[0], -1)) for x in spectra]


def _rolled(x, t):
    """x at the neighbour of tap t, zero beyond the ends of y."""
    dy, dz, dx = t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1
    y = torch.roll(x, (-dz, -dx), (1, 2))
    out = torch.zeros_like(y)
    n = y.shape[0]
    out[max(0, -dy):n - max(0, dy)] = y[max(0, dy):n - max(0, -dy)]
    return out


def _exact_net(c, seed):
    bf = lambda a: torch.from_numpy(a).to(DEV).to(torch.bfloat16).double()  # noqa: E731
    params = [(bf(w), torch.from_numpy(b).to(DEV).double()) for w, b in _net_params(seed)]
    x, base, target = _net_input(c["Y"], c["Z"], c["X"], seed)

    def conv(i, h):
        w, b = params[i]
        return sum(_rolled(h, t) @ w[t].T for t in range(27)) + b

    last = len(params) - 1
    acts, h = [x.double()], conv(0, x.double())
    acts.append(h)
    for i in range(1, last, 2):
        t = conv(i, h).clamp(min=0.0)
        h = h + conv(i + 1, t)
        acts += [t, h]
    corr = conv(last, h)
    if c["kind"] == "infer":
        return corr
    nvox = base.shape[0]
    diff = base.double() + corr.reshape(nvox, -1)[:, :3] - target.double()
    d = torch.zeros_like(corr)
    d[..., :3] = (2.0 / (3 * nvox) * diff).reshape(d.shape[:3] + (3,))
    grads = [None] * len(params)

    def back(i, h, dy, down=True):
        w, b = params[i]
        flat = dy.reshape(-1, dy.shape[-1])
        gw = torch.stack([flat.T @ _rolled(h, t).reshape(flat.shape[0], -1) for t in range(27)])
        grads[i] = torch.cat([gw.reshape(-1), flat.sum(0)])
        return sum(_rolled(dy, 26 - t) @ w[t] for t in range(27)) if down else None

    d = back(last, acts[-1], d)
    for i in range(last - 2, 0, -2):
        t = acts[i + 1]
        d = d + back(i, acts[i], back(i + 1, t, d) * (t > 0))
    back(0, acts[0], d, down=False)
    return {"corr": corr, "loss": (diff ** 2).mean().reshape(1), "grad": torch.cat(grads), "master": None}


def exact(case, seed):
    c = case
    if c["kind"] in ("train", "infer"):
        return _exact_net(c, seed)
    if c["ngalx2"]:
        return None  # the bands' columns of unlike length take far longer than the step itself
    if c["kind"] == "ensemble":
        return [_Exact(c, seed, m).step(c["steps"]) for m in range(c["members"])]
    e = _Exact(c, seed)
    fields = e.step(c["steps"])
    if c["kind"] == "step":
        return fields
    stats, cond, spectra = e.statistics()
    return {"fields": fields, "mpgx": e.mpgx, "Qx": e.flow(), "dt": e.cfl(), "stats": stats, "cond": cond, "spectra": spectra}
