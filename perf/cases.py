"""Timed workloads of the 2.5D FDTD vocal-tract solver, through its public Python handles.

A case is one of four kinds of call a program makes:

  run      a solver or batch that is kept; every pass restarts it and advances it `steps` time steps
  oneshot  area functions in host memory to traces in host memory: create the batch, run it, close it
  grad     checkpointed forward and reverse-time adjoint of a kept batch, for a given dL/dtrace
  post     formants and audio samples of listener traces that are on the GPU

Tubes are seeded smooth random area functions over the ranges of the synthetic workloads (12-20 cm long,
2-4 cm wide, 44 sections, and the uniform 17.5 x 3 cm tube).  `exact` restates the discrete system here in
64 bits (maps, step, two-mass source, adjoint, formants, audio filter), in numpy and torch.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "vocalsim-2p5d-fdtd_b200" / "python"))

import vocalsim_b200 as V                                     # noqa: E402
from vocalsim_b200.audio import audio                         # noqa: E402
from vocalsim_b200.spectrum import formants                   # noqa: E402

SECTIONS = 44
CKPT = 512
F32 = np.float32


# ---- the cases -------------------------------------------------------------------------------------------

def case(name=None, kind="run", tubes=1, steps=33075, fast=1, source="gauss", shape=2, mouth=0, mul=15, tube="vowel"):
    c = dict(kind=kind, tubes=tubes, steps=steps, fast=fast, source=source, shape=shape, mouth=mouth, mul=mul, tube=tube)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a few milliseconds of sound from a tube that is being edited interactively: launches and latency count
        case("chunk_single", steps=512, tube="uniform", shape=1),
        # the uniform 17.5 x 3 cm circular tube for 50 ms: the transfer function of one tube
        case("single_uniform", tube="uniform", shape=1),
        # the same length of a vowel tube in the default, reference arithmetic (a drop-in use of the library)
        case("single_exact", fast=0, steps=16537),
        # 100 ms of voiced sound: the two-mass glottal source (double model) on a vowel tube
        case("voiced_single", source="tmm64", steps=66150),
        # the reference's float two-mass model in the reference arithmetic, closed (Dirichlet) mouth
        case("voiced_exact", source="tmm", fast=0, steps=8192, mouth=1),
        # a handful of tubes stepped together (one speaker's vowels)
        case("batch_5", tubes=5, steps=16384),
        # a medium batch of circular tubes in the reference arithmetic, sine source
        case("batch_48_exact", tubes=48, steps=8192, fast=0, source="sine", shape=1),
        # 256 tubes for 50 ms: the batched-forward workload
        case("batch_256", tubes=256),
        # area functions in, traces out, nothing kept: 96 tubes for 10 ms
        case("oneshot_96", kind="oneshot", tubes=96, steps=6615),
        # the gradient of one voiced vowel tube over 20 ms
        case("grad_voiced", kind="grad", source="tmm64", steps=13230),
        # the gradient of the inversion's batch: 64 tubes on the finer grid, a part of its 20 ms
        case("grad_64_fine", kind="grad", tubes=64, steps=4096, mul=30),
        # formants and audio of a batch's 50 ms traces
        case("post_256", kind="post", tubes=256),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "oneshot", "grad", "grad", "post"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    tubes = log(1, 256)
    fast = rng.choice([1, 1, 0])
    source = rng.choice(["gauss", "gauss", "sine"] + (["tmm", "tmm64"] if tubes <= 8 else []))
    c = case(kind=kind, tubes=tubes, fast=fast, shape=rng.choice([1, 2]), mouth=rng.choice([0, 0, 1]), source=source)
    if kind == "grad":
        c["mul"] = rng.choice([15, 30])
        c["tubes"] = min(tubes, 64)
        c["source"] = "gauss" if c["tubes"] > 2 else source
        c["steps"] = log(512, min(8192, 64 * 4096 // c["tubes"]))
    elif kind == "post":
        c["steps"] = log(4001, 66150)
        c["tubes"] = min(tubes, 256 * 33075 // c["steps"])
        c["source"] = "gauss"
    else:
        c["steps"] = log(256, min(66150, 256 * 33075 // (tubes * (3 if not fast else 1))))
        if tubes <= 16 and rng.random() < 0.3:
            c["mul"] = 30
    return c


# ---- inputs ----------------------------------------------------------------------------------------------

def tubes_of(c, seed):
    """(section lengths cm, areas cm^2) of every tube, float32.  Lengths and greatest widths belong to the
    case (they fix the frames), the area curves and the uniform tube come from the seed."""
    size = np.random.default_rng([c["tubes"], c["mul"], 70])
    rng = np.random.default_rng([seed, 71])
    out = []
    for _ in range(c["tubes"]):
        length = size.uniform(12.0, 20.0) if c["tubes"] > 1 else 17.5
        # the widest section of a batch's tube is 2-4 cm across (3:1 ellipse)
        wide = size.uniform(2.0 if c["mul"] <= 15 else 3.0, 4.0) if c["tubes"] > 1 else 3.9
        most = 3.0 * math.pi * (wide / 6.0) ** 2
        if c["tube"] == "uniform":
            length += rng.uniform(-0.5, 0.5)
            out.append((np.array([length], F32), np.array([math.pi * rng.uniform(1.3, 1.7) ** 2], F32)))
            continue
        k = np.arange(1, 6)
        amp = rng.uniform(-1.5, 1.5, size=5) / np.sqrt(k)
        phase = rng.uniform(0.0, 2.0 * np.pi, size=5)
        x = (np.arange(SECTIONS) + 0.5) / SECTIONS
        a = 2.2 + (amp * np.cos(np.pi * k * x[:, None] + phase)).sum(axis=1)
        a = np.clip(a, 0.3, 5.0)
        # below about 1 cm^2 the scheme itself is unstable on the finer grid
        a = np.maximum(a * (most / a.max()), 0.0 if c["mul"] <= 15 else 1.2)
        out.append((np.full(SECTIONS, length / SECTIONS, F32), a.astype(F32)))
    return out


def seed_gradient(c, seed):
    """dL/dtrace of the grad cases: a smooth residual, as a spectral loss gives."""
    rng = np.random.default_rng([seed, 72])
    t = np.arange(c["steps"]) / (44100.0 * c["mul"])
    f = rng.uniform(200.0, 5000.0, size=(c["tubes"], 6, 1))
    a = rng.standard_normal((c["tubes"], 6, 1))
    return (1e-3 * a * np.cos(2 * np.pi * f * t + rng.uniform(0, 6.28, f.shape))).sum(axis=1).astype(F32)


def listener_traces(c, seed):
    """Traces as a tube's listener gives them: decaying resonances (formants) with a little noise."""
    rng = np.random.default_rng([seed, 73])
    g = torch.Generator(device="cuda").manual_seed(seed)
    fs = 44100.0 * c["mul"]
    t = torch.arange(c["steps"], device="cuda", dtype=torch.float64) / fs
    x = torch.zeros((c["tubes"], c["steps"]), dtype=torch.float64, device="cuda")
    for lo, hi in ((300, 900), (1000, 2200), (2400, 3100), (3300, 4200), (4400, 5000)):
        f = torch.from_numpy(rng.uniform(lo, hi, (c["tubes"], 1))).cuda()
        b = torch.from_numpy(rng.uniform(60, 160, (c["tubes"], 1))).cuda()
        a = torch.from_numpy(rng.uniform(0.3, 1.0, (c["tubes"], 1))).cuda()
        x += a * torch.exp(-math.pi * b * t) * torch.sin(2 * math.pi * f * t)
    x += 1e-4 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
    return (40.0 * x).to(torch.float32)


def params(c):
    src = {"gauss": V.SRC_GAUSS, "sine": V.SRC_SINE, "tmm": V.SRC_TMM, "tmm64": V.SRC_TMM}[c["source"]]
    return V.params(num_steps=c["steps"], fast_math=c["fast"], cross_sectional_shape=c["shape"], srate_mul=c["mul"],
                    mouth_radiation_cond=c["mouth"], source_type=src, tmm_f64=int(c["source"] == "tmm64"),
                    tmm_ps_pa=800.0)


def prepare(c, seed):
    if c["kind"] == "post":
        return dict(case=c, traces=listener_traces(c, seed))
    geoms = [V.Geometry(*t) for t in tubes_of(c, seed)]
    ps = [params(c) for _ in geoms]
    s = dict(case=c, params=ps, geoms=geoms)
    if c["kind"] == "grad":
        s.update(handle=V.Batch(ps, geoms), seed_gradient=seed_gradient(c, seed))
    elif c["kind"] == "run" and c["tubes"] == 1:
        s.update(handle=V.Solver(ps[0], geoms[0]))
    elif c["kind"] == "run":
        s.update(handle=V.Batch(ps, geoms),
                 traces=torch.empty((c["tubes"], c["steps"]), dtype=torch.float32, device="cuda"))
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "run":
        h = s["handle"]
        h.reset()
        if c["tubes"] == 1:
            return h.run(c["steps"])
        h.run_device(c["steps"], s["traces"].data_ptr())
        return s["traces"]
    if c["kind"] == "oneshot":
        b = V.Batch(s["params"], s["geoms"])
        tr = b.run(c["steps"])
        b.close()
        return tr
    if c["kind"] == "grad":
        tr = s["handle"].forward_ckpt(c["steps"], CKPT)
        maps, gz = s["handle"].adjoint(s["seed_gradient"])
        # the tubes' frames are views of one array per map
        return {"trace": tr, "maps": [g.base for g in maps[0]], "z_inv": gz}
    return {"formants": formants(s["traces"], 44100.0 * c["mul"]), "audio": audio(s["traces"], c["mul"])}


# ---- the work a pass cannot do without -------------------------------------------------------------------

def frame(c, lengths, areas):
    """Frame rows and columns of a tube."""
    k = physics(c["mul"])
    width, _ = widths(c, areas)
    cells = [odd_cells(w, k["ds"]) for w in width]
    L = half_up(float(sum_f32(lengths * F32(1e-2)) / k["ds"]))
    mic = half_up(float(F32(3) * F32(1e-3) / k["ds"]))
    return max(cells) + 16, (L + 2 if c["mouth"] else L + 1 + mic) + 14


def work(c):
    """A whole run keeps a tube's state on the chip at best: maps and source in, traces out.  The operations
    are the update's: 8 for a pressure, 5 for each of two velocities, per cell and step (an adjoint
    recomputes the forward and does about the same twice over)."""
    n, steps = c["tubes"], c["steps"]
    if c["kind"] == "post":
        return {"bytes": 4.0 * n * steps * (1 + 1 / c["mul"]), "flops": n * steps * (10.0 + 2.5 * math.log2(steps))}
    cells = 0
    for lengths, areas in tubes_of(c, 1):
        h, w = frame(c, lengths, areas)
        cells += (h - 2) * (w - 2)
    up = 18.0 * cells * steps
    if c["kind"] == "grad":
        # 18 floats per cell of state, maps and gradients, and the traces both ways
        return {"bytes": 4.0 * (n * steps * 2 + cells * 18), "flops": 4.0 * up}
    return {"bytes": 4.0 * (n * steps * (1 + (c["source"] in ("gauss", "sine")) / n) + cells * 6), "flops": up}


# ---- the discrete system in 64 bits ----------------------------------------------------------------------
# The grid is the reference's: its float32 rounding decides which cells are walls and what the depths are,
# so the maps are built in float32 and everything that is stepped on them is float64.

WALL, AIR, EXC, PML0, PML5, DEAD, NOPRES = 0, 1, 2, 3, 8, 10, 11


def half_up(x):
    return int(math.floor(x + 0.5))


def sum_f32(v):
    t = F32(0)
    for x in v:
        t = F32(t + x)
    return t


def physics(mul):
    c, rho = F32(350), F32(1.14)
    dt = F32(1) / F32(44100 * mul)
    ds = F32(F32(dt * c) * np.sqrt(F32(2)))
    kappa = F32(F32(rho * c) * c)
    return dict(c=c, rho=rho, dt=dt, ds=ds, K1=float(F32(kappa * dt) / ds), b=float(dt / F32(rho * ds)))


def widths(c, areas):
    a = areas * F32(1e-2) * F32(1e-2)
    if c["shape"] == 1:
        return (2.0 * np.sqrt(a.astype(np.float64) / math.pi)).astype(F32), np.zeros(len(a), F32)
    lx = np.sqrt((a.astype(np.float64) / (3.0 * math.pi)).astype(F32))
    return lx * F32(6), lx * F32(2)


def odd_cells(w, ds):
    x = F32(w / ds)
    n = half_up(float(x))
    n += n == 0
    if n % 2 == 0:
        n += -1 if F32(n) - x > 0 else 1
    return n


def maps(c, lengths, areas):
    """Cell types, z_inv flags, depths (float64 values of the float32 maps) and marked cells of one tube."""
    k = physics(c["mul"])
    ds = k["ds"]
    width, minor = widths(c, areas)
    cells = [odd_cells(w, ds) for w in width]
    H, W = frame(c, lengths, areas)
    lm = lengths * F32(1e-2)
    L = half_up(float(sum_f32(lm) / ds))
    sx, my = 8, int(math.ceil(H / 2.0)) - 1
    ex = sx + L - 1
    cum = [sum_f32(lm[:i + 1]) for i in range(len(lm))]
    typ = np.full((H, W), AIR)
    seg = np.zeros((H, W), bool)
    up, down, sec = [], [], []
    for i in range(L):
        x = F32(F32(i + 1) * ds)
        s = 0
        while s < len(lm) - 1 and x > F32(cum[s] + F32(ds * F32(0.5))):
            s += 1
        r = (cells[s] - 1) // 2
        up.append(my - r - 1)
        down.append(my + r + 1)
        sec.append(s)
        for row in (up[i], down[i]):
            typ[row, sx + i], seg[row, sx + i] = WALL, True
    for i in range(1, L - 1):
        jump = up[i] - up[i - 1]
        if abs(jump) > 1:
            col = i if jump > 1 else i - 1
            lo, hi = sorted((up[i], up[i - 1])), sorted((down[i], down[i - 1]))
            for a, b in (lo, hi):
                typ[a:b + 1, sx + col], seg[a:b + 1, sx + col] = WALL, True
    typ[up[0] + 1:down[0], sx - 1] = EXC
    typ[up[0], sx - 1] = typ[down[0], sx - 1] = WALL
    mic = half_up(float(F32(3) * F32(1e-3) / ds))
    if c["mouth"]:
        typ[up[-1]:down[-1] + 1, ex + 1] = NOPRES
    lis = (my, ex - mic if c["mouth"] else ex + 3 + mic)
    dX, dY = np.full((H, W), F32(0.5)), np.full((H, W), F32(0.5))
    for i in range(L):
        x, air = sx + i, down[i] - up[i] - 1
        h = int(math.ceil(air * 0.5)) - 1
        if c["shape"] == 1:
            r = F32(F32(F32(air) / F32(2)) * ds)
            r2 = F32(r * r)
            rad = lambda y: F32(float(r2) - float(y) * float(y))     # one rounding, as a fused multiply-add
        else:
            a = F32(F32(F32(air) * ds) / F32(2))
            hb = F32(minor[sec[i]] / F32(2))
            a2, b2 = F32(a * a), F32(hb * hb)
            rad = lambda y: F32(b2 * F32(F32(1) - F32(F32(y * y) / a2)))
        for q in range(h, -1, -1):
            depth = lambda y: F32(F32(2) * np.sqrt(rad(F32(F32(y) * ds))))
            ru, rl = up[i] + (h - q) + 1, down[i] - (h - q) - 1
            dX[ru, x] = dX[rl, x] = depth(q)
            dY[ru, x] = depth(q + 0.5) if q != h else F32(0)
            dY[rl, x] = depth(q - 0.5)
        for row in (up[i], down[i]):
            dX[row, x] = dY[row, x] = F32(0)
    for d in (dX, dY):
        d[d == F32(0.5)] = d[my, ex]
    h5 = F32(0.5)
    xs = h5 * (dX + np.concatenate([dX[:, 1:], np.full((H, 1), dX[my, ex])], 1))
    ys = h5 * (dY + np.concatenate([np.full((1, W), dY[my, ex]), dY[:-1]], 0))
    left = np.concatenate([np.full((H, 1), xs[my, ex]), xs[:, :-1]], 1)
    below = np.concatenate([ys[1:], np.full((1, W), ys[my, ex])], 0)
    dP = F32(0.25) * (((xs + ys) + left) + below)
    typ[0], typ[-1], typ[:, 0], typ[:, -1] = DEAD, DEAD, DEAD, DEAD
    for l in range(6):
        typ[1 + l, 1 + l:W - 1 - l] = typ[H - 2 - l, 1 + l:W - 1 - l] = PML5 - l
    for l in range(6):
        typ[1 + l:H - 1 - l, 1 + l] = typ[1 + l:H - 1 - l, W - 2 - l] = PML5 - l
    mu2 = F32(float(F32(0.025)) * (math.pi / float(F32(1.84))))
    alpha = F32(1) / (F32(0.5) + F32(0.25) * (mu2 + F32(1) / mu2))
    q = np.sqrt(F32(1) - alpha)
    z = F32(1) / (k["rho"] * k["c"] * ((F32(1) + q) / (F32(1) - q)))
    floor = lambda d: np.maximum(d, F32(0.001)).astype(np.float64)
    return dict(type=typ, seg=seg, dP=floor(dP), dX=floor(xs), dY=floor(ys), lis=lis, exc=(my, sx - 1), z=float(z),
                H=H, W=W)


class System:
    """The step of all tubes of a case as float64 tensors over one padded frame, and its transpose."""

    def __init__(self, c, seed, device):
        self.c, self.dev = c, device
        k = physics(c["mul"])
        self.K1, self.b, self.dt = k["K1"], k["b"], k["dt"]
        ms = [maps(c, *t) for t in tubes_of(c, seed)]
        self.n, self.ms = len(ms), ms
        H, W = max(m["H"] for m in ms), max(m["W"] for m in ms)
        full = lambda v: np.full((self.n, H, W), v)
        typ, seg = full(DEAD), full(False)
        dP, dX, dY = full(1.0), full(1.0), full(1.0)
        for i, m in enumerate(ms):
            s = (i, slice(0, m["H"]), slice(0, m["W"]))
            typ[s], seg[s], dP[s], dX[s], dY[s] = m["type"], m["seg"], m["dP"], m["dX"], m["dY"]
        beta = np.isin(typ, [AIR, NOPRES] + list(range(PML0, PML5 + 1))).astype(float)
        sig = np.zeros(typ.shape)
        sig[(typ == WALL) | (typ == EXC)] = float(self.dt)
        sig[typ == DEAD] = 1e6
        for l in range(6):
            sig[typ == PML0 + l] = float(F32(F32(l) / F32(5)) * F32(0.5))
        right = lambda a, v: np.concatenate([a[:, :, 1:], np.full((self.n, H, 1), v)], 2)
        top = lambda a, v: np.concatenate([np.full((self.n, 1, W), v), a[:, :-1]], 1)
        zi = np.array([m["z"] for m in ms])[:, None, None] * (seg & True)
        exc = (typ == EXC).astype(float)
        inner = np.zeros(typ.shape)
        for i, m in enumerate(ms):
            inner[i, 1:m["H"] - 1, 1:m["W"] - 1] = 1.0

        def direction(nb, other, weight):
            bn, bo, en = nb(beta, 0.0), other(beta, 0.0), nb(exc, 0.0)
            mS, mB = np.maximum(sig, nb(sig, 1e6)), beta * bn
            g = inner / (mB + mS)
            n = 1.0 - np.maximum(exc, en)
            nout = np.where(bo == 0, float(F32(0.707106)), 1.0)
            out, inn = beta * (1 - bn) * nout * n * mS * g, bn * (1 - beta) * n * mS * g
            return dict(al=mB * g, pc=mB * g * self.b, zo=out * (seg & True), zi=inn * (seg & True), ce=weight * exc * mS * g)

        x = direction(right, top, 1.0)
        y = direction(top, right, 0.0)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)
        z = np.array([m["z"] for m in ms])[:, None, None]
        self.ax, self.bx = t(x["pc"] + x["zo"] * z), t(x["pc"] + x["zi"] * z)
        self.ay, self.by = t(y["pc"] + y["zo"] * z), t(y["pc"] + y["zi"] * z)
        self.alx, self.aly, self.ce = t(x["al"]), t(y["al"]), t(x["ce"])
        self.zox, self.zix, self.zoy, self.ziy = t(x["zo"]), t(x["zi"]), t(y["zo"]), t(y["zi"])
        s1 = 1.0 + sig
        live = inner * (typ != NOPRES if c["mouth"] else np.ones(typ.shape))
        self.g, self.kd = t(live / s1), t(live * self.K1 / (s1 * dP))
        self.dP, self.dX, self.dY, self.inner = t(dP), t(dX), t(dY), t(inner)
        self.shape = typ.shape
        self.rows = torch.arange(self.n, device=device)
        at = lambda key: tuple(torch.tensor([m[key][j] for m in ms], device=device) for j in (0, 1))
        self.lis, self.exc = at("lis"), at("exc")

    def zeros(self):
        return [torch.zeros(self.shape, dtype=torch.float64, device=self.dev) for _ in range(3)]

    def divergence(self, X, Y):
        U, Wy = X * self.dX, Y * self.dY
        S = U + Wy
        S[:, :, 1:] -= U[:, :, :-1]
        S[:, :-1] -= Wy[:, 1:]
        return S

    def step(self, s, e):
        """s = [P, Vx, Vy] in place; e = the excitation velocity."""
        P, X, Y = s
        S = self.divergence(X, Y)
        P.mul_(self.g).addcmul_(self.kd, S, value=-1.0)
        X.mul_(self.alx).addcmul_(self.ax, P)
        X[:, :, :-1].addcmul_(self.bx[:, :, :-1], P[:, :, 1:], value=-1.0)
        X.add_(self.ce * e)
        Y.mul_(self.aly).addcmul_(self.ay, P)
        Y[:, 1:].addcmul_(self.by[:, 1:], P[:, :-1], value=-1.0)

    def source(self, steps):
        i = np.arange(steps)
        t = (i * float(self.dt)).astype(F32)
        if self.c["source"] == "sine":
            return 25.0 * np.sin(2 * math.pi * 440.0 * t.astype(np.float64))
        peak = F32(0.646) / F32(1e4)
        e = ((t - peak) / F32(F32(0.29) * peak)).astype(np.float64)
        return float(F32(0.025)) * np.exp(-e * e)

    def forward(self, s, start, count, trace, e):
        for n in range(start, start + count):
            self.step(s, e[n])
            if trace is not None:
                trace[:, n] = s[0][self.rows, self.lis[0], self.lis[1]]

    def traces(self, steps):
        s = self.zeros()
        tr = torch.zeros((self.n, steps), dtype=torch.float64, device=self.dev)
        if self.c["source"].startswith("tmm"):
            model = [TwoMass(800.0, self.c["mul"]) for _ in range(self.n)]
            e = torch.zeros((self.n, 1, 1), dtype=torch.float64, device=self.dev)
            for n in range(steps):
                p = s[0][self.rows, self.exc[0], self.exc[1]].tolist()
                for i, m in enumerate(model):
                    e[i] = m.step(p[i])
                self.step(s, e)
                tr[:, n] = s[0][self.rows, self.lis[0], self.lis[1]]
            return tr
        self.forward(s, 0, steps, tr, self.source(steps).tolist())
        return tr

    def gradients(self, steps, seed):
        """Traces, and dL/d(dP, dX, dY, z) for dL/dtrace = seed (n x steps), by the transposed step."""
        e = self.source(steps).tolist()
        s, marks = self.zeros(), []
        tr = torch.zeros((self.n, steps), dtype=torch.float64, device=self.dev)
        for k in range(0, steps, CKPT):
            marks.append([v.clone() for v in s])
            self.forward(s, k, min(CKPT, steps - k), tr, e)
        lP, lX, lY = self.zeros()
        gP, gX, gY = self.zeros()
        gz = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
        rd = self.kd / self.dP
        for k in range((steps - 1) // CKPT * CKPT, -1, -CKPT):
            s, hist = marks.pop(), []
            for n in range(k, min(k + CKPT, steps)):
                hist.append([v.clone() for v in s])
                self.step(s, e[n])
            hist.append(s)
            for n in range(min(k + CKPT, steps) - 1, k - 1, -1):
                P1, (_, X, Y) = hist[n + 1 - k][0], hist[n - k]
                gz.addcmul_(lX, self.zox * P1).addcmul_(lY, self.zoy * P1)
                gz[:, :, :-1].addcmul_(lX[:, :, :-1], self.zix[:, :, :-1] * P1[:, :, 1:], value=-1.0)
                gz[:, 1:].addcmul_(lY[:, 1:], self.ziy[:, 1:] * P1[:, :-1], value=-1.0)
                mu = lP + self.ax * lX + self.ay * lY
                mu[:, :, 1:] -= (self.bx * lX)[:, :, :-1]
                mu[:, :-1] -= (self.by * lY)[:, 1:]
                mu[self.rows, self.lis[0], self.lis[1]] += seed[:, n]
                gP.addcmul_(mu * rd, self.divergence(X, Y))
                q = mu * self.kd
                lU, lW = -q, -q
                lU[:, :, :-1] += q[:, :, 1:]
                lW[:, 1:] += q[:, :-1]
                lP = mu * self.g
                gX.addcmul_(X, lU)
                gY.addcmul_(Y, lW)
                lX = (self.alx * lX + self.dX * lU) * self.inner
                lY = (self.aly * lY + self.dY * lW) * self.inner
            del hist
        return tr, gP, gX, gY, gz.sum((1, 2))


class TwoMass:
    """The Ishizaka-Flanagan two-mass model, one tube."""

    def __init__(self, ps, mul):
        cm, gram, dyn = float(F32(1e-2)), float(F32(1e-3)), float(F32(1e-5))
        f = lambda v: float(F32(v))
        self.ps, self.sr = ps, 44100.0 * mul
        self.mu, self.rho = 1.86e-4 * float(F32(dyn) / (F32(cm) * F32(cm))), 1.14
        self.m = f(0.125) * gram, f(0.025) * gram
        self.d = f(0.25) * cm, f(0.05) * cm
        self.k = 80000.0 * (dyn / cm), 8000.0 * (dyn / cm)
        self.kc, self.eta, self.etah = 25000.0 * (dyn / cm), 100.0 / (cm * cm), 500.0 / (cm * cm)
        self.a0, self.lg, self.A1 = f(0.05) * cm * cm, f(1.4) * cm, 3.0 * cm * cm
        root = [math.sqrt(a * b) for a, b in zip(self.k, self.m)]
        self.ro = 2 * f(0.2) * root[0], 2 * f(0.6) * root[1]
        self.rc = 2 * f(1.1) * root[0], 2 * f(1.9) * root[1]
        self.x, self.xo, self.ug, self.ugo = [0.0, 0.0], [0.0, 0.0], 0.0, 0.0

    def step(self, p1):
        d, lg, rho, ps, sr, x, ug = self.d, self.lg, self.rho, self.ps, self.sr, self.x, self.ug
        A = [self.a0 + 2 * lg * v for v in x]
        c12 = 12 * self.mu * lg * lg
        Rv, Lg = [c12 * d[i] / A[i] ** 3 for i in (0, 1)], [rho * d[i] / A[i] for i in (0, 1)]
        g, du = self.a0 / (2 * lg), ug - self.ugo
        open_ = [v > -g for v in x]
        pm1 = ps
        if all(open_):
            pm1 = ps - 1.37 * (rho / 2) * (ug / A[0]) ** 2 - 0.5 * (Rv[0] * ug + Lg[0] * sr * du)
        pm2 = 0.0
        if open_[0]:
            pm2 = ps
            if open_[1]:
                pm2 = (pm1 - (0.5 * (Rv[0] + Rv[1]) * ug + (Lg[0] + Lg[1]) * du * sr)
                       - (rho / 2) * ug * ug * (1 / A[1] ** 2 - 1 / A[0] ** 2))
        F = [pm1 * d[0] * lg, pm2 * d[1] * lg]
        a, b = [0.0, 0.0], [0.0, 0.0]
        for i in (0, 1):
            shut = x[i] + g < 0
            h, r = (3 * self.k[i], self.rc[i]) if shut else (0.0, self.ro[i])
            a[i] = (self.k[i] + h + self.kc) / sr ** 2 + r / sr + self.m[i]
            sp = self.k[i] * self.eta * x[i] ** 3 + h * (g + self.etah * (g + x[i]) ** 3)
            b[i] = (2 * self.m[i] + r / sr) * x[i] - self.m[i] * self.xo[i] + (F[i] - sp) / sr ** 2
        off = -self.kc / sr ** 2
        det = a[0] * a[1] - off * off
        new = [(a[1] * b[0] - off * b[1]) / det, (a[0] * b[1] - off * b[0]) / det]
        A = [self.a0 + 2 * lg * v for v in new]
        u = 0.0
        if min(A) >= 0:
            r = A[1] / self.A1
            R = ((rho / 2) * abs(ug) * (0.37 / A[0] ** 2 + (1 - 2 * r * (1 - r)) / A[1] ** 2)
                 + c12 * (d[0] / A[0] ** 3 + d[1] / A[1] ** 3))
            Lt = rho * (d[0] / A[0] + d[1] / A[1])
            u = ((ps - p1) / sr + Lt * ug) / (R / sr + Lt)
        self.xo, self.x, self.ugo, self.ug = x, new, ug, u
        return u


def exact_post(c, seed):
    x = listener_traces(c, seed).double()
    fs = 44100.0 * c["mul"]
    level = (10 * torch.log10(torch.fft.fft(x).abs() ** 2)).cpu().numpy()
    n, out = c["steps"], np.zeros((c["tubes"], 3, 4))
    freq = np.linspace(0.0, fs, n)
    for t, v in enumerate(level):
        i, found = 1, 0
        while found < 4 and i < n - 1:
            if not (v[i] > v[i - 1] and v[i] > v[i + 1]):
                i += 1
                continue
            cut, lo, hi = v[i] - 3, i, i
            while lo > 0 and v[lo] > cut:
                lo -= 1
            while hi < n - 1 and v[hi] > cut:
                hi += 1
            f_lo = np.interp(cut, [v[lo], v[lo + 1]], [freq[lo], freq[lo + 1]])
            f_hi = np.interp(cut, [v[hi - 1], v[hi]], [freq[hi - 1], freq[hi]])
            out[t, :, found] = f_hi - f_lo, freq[i], v[i]
            found, i = found + 1, hi
    a = (x / x.abs().amax(1, keepdim=True)).clip(-1, 1).cpu().numpy()
    if c["mul"] > 1:
        # 2nd-order Butterworth low-pass at 5050 Hz by the bilinear transform
        w = math.tan(math.pi * 5050.0 / fs)
        n0 = 1 + math.sqrt(2) * w + w * w
        b0, a1, a2 = w * w / n0, 2 * (w * w - 1) / n0, (1 - math.sqrt(2) * w + w * w) / n0
        y, z0, z1 = np.zeros_like(a), np.zeros(len(a)), np.zeros(len(a))
        for i in range(n):
            u = a[:, i]
            y[:, i] = b0 * u + z0
            z0 = z1 + 2 * b0 * u - a1 * y[:, i]
            z1 = b0 * u - a2 * y[:, i]
        a = y[:, ::c["mul"]]
    return {"formants": out, "audio": a}


def exact(c, seed):
    if c["kind"] == "post":
        return exact_post(c, seed)
    voiced = c["source"].startswith("tmm")
    # a self-oscillating source leaves a 64-bit run's path after some ten thousand steps whatever is done
    # in 32 bits, and the float model earlier; the sizes below take about 20 seconds
    if voiced and (c["tubes"] * c["steps"] > 40000 or c["kind"] == "grad" or c["source"] == "tmm"):
        return None
    s = System(c, seed, "cpu" if voiced and c["tubes"] == 1 else "cuda")
    cells = float(np.prod(s.shape))
    cost = c["steps"] * max(110e-6, cells * 1.3e-10) * (5 if c["kind"] == "grad" else 1)
    if cost > 20.0 or (c["kind"] == "grad" and cells * 24 * (CKPT + c["steps"] / CKPT) > 9e10):
        return None
    if c["kind"] != "grad":
        tr = s.traces(c["steps"]).cpu().numpy()
        return tr[0] if c["kind"] == "run" and c["tubes"] == 1 else tr
    seedg = torch.from_numpy(seed_gradient(c, seed)).double().cuda()
    tr, gP, gX, gY, gz = s.gradients(c["steps"], seedg)
    cut = lambda g: np.concatenate([g[i, :m["H"], :m["W"]].cpu().numpy().ravel() for i, m in enumerate(s.ms)])
    return {"trace": tr.cpu().numpy(), "maps": [cut(g) for g in (gP, gX, gY)], "z_inv": gz.cpu().numpy()}
