"""Performance cases of the flow solver: what users of the framework have it do.

A case is one of four uses of the public API (canard_b200.api), over the grids
and boundary set-ups of canard_b200.cases:

* ``run``: a time-stepping run from an initial state: set the time and the
  state of every block, ``step(n)``, read the state back.
* ``record``: the same run the way the reference's program drives it
  (canard_b200.driver): after every step the time-averaged recording advances
  and the time is read; at the end the FP32 output fields are taken. This is how
  a mixed-precision run is used; an FP64 run also reads its final state.
* ``host``: steps through host memory (``step_host``), for a program that owns
  the state on the host between steps.
* ``operators``: the drop-in derivative and filter calls on host arrays.

All host arrays that take part in a pass are pinned, as a program that moves
its state every run keeps them. ``exact`` is the same scheme in 64 bits, with
the compact operators as dense matrices.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from canard_b200 import api, cases

PRECISION = {"fp64": api.FP64, "fast": api.FP64_FAST, "mixed": api.FP32_MIXED}
GAM, PRNDTL = 1.4, 0.71
STEPS = 20


def listed():
    def case(name, use, flow, size, precision="fp64", viscous=1, steps=STEPS, count=1, layout=0):
        return {"name": name, "use": use, "flow": flow, "nx": size[0], "ny": size[1], "nz": size[2],
                "precision": precision, "viscous": viscous, "steps": steps, "count": count, "layout": layout}
    return [
        # the smallest complete run: the reference's validation block through its program's loop
        case("validation 50x50x16 driver", "record", "validation", (50, 50, 16)),
        # many small blocks with straight interfaces: the reference's toy set-up
        case("toy 6x100x100x16", "run", "toy", (100, 100, 16)),
        # the 64^3 Taylor-Green run, the smallest benchmark configuration: launches and latency count
        case("tgv 64 fp64", "run", "tgv", (64, 64, 64)),
        # ordinary odd, uneven sides; inviscid
        case("tgv 95x77x61 inviscid fast", "run", "tgv", (95, 77, 61), "fast", viscous=0),
        # the benchmark block in its three precisions
        case("tgv 256 fp64", "run", "tgv", (256, 256, 256)),
        case("tgv 256 fast", "run", "tgv", (256, 256, 256), "fast"),
        case("tgv 256 mixed driver", "record", "tgv", (256, 256, 256), "mixed"),
        # curvilinear multi-block run: interfaces, characteristic boundaries, sponge
        case("curv 4x192x128x64", "run", "curv", (192, 128, 64)),
        # the vortex through an outflow of the accuracy study, mixed precision
        case("vortex 384x256x128 mixed", "record", "vortex", (384, 256, 128), "mixed"),
        # 64 independent uneven cases advanced together (a parameter study)
        case("batch of 64 mixed", "record", "batch", (64, 64, 64), "mixed", count=64, layout=11),
        # a coupled program that owns the state on the host between steps
        case("host-owned tgv 128 fast", "host", "tgv", (128, 128, 128), "fast", steps=10),
        # drop-in operator calls on host arrays
        case("operators 120x96x80", "operators", "tgv", (120, 96, 80)),
    ]


def draw(rng):
    """A case of the same ranges: sides 24..288 cells (uneven, odd and even), at most
    the points of the largest listed block, any use, flow and precision."""
    use = rng.choice(["run", "run", "record", "record", "host", "operators"])
    flow = "tgv" if use in ("host", "operators") else rng.choice(["tgv", "tgv", "vortex", "curv", "validation",
                                                                   "toy", "batch"])
    precision = rng.choice(["fp64", "fast", "mixed"])
    if precision == "mixed" and use == "run":
        use = "record"
    if precision == "mixed" and use in ("host", "operators"):
        precision = "fp64"
    blocks = {"curv": 4, "toy": 6}.get(flow, 1)
    while True:
        n = [int(round(math.exp(rng.uniform(math.log(24), math.log(288))))) for _ in range(3)]
        most = 3e6 if use in ("host", "operators") else 1.6e7
        if blocks * n[0] * n[1] * n[2] <= most:
            break
    count, layout = 1, 0
    if flow == "batch":
        n, count, layout = [64, 64, 64], rng.randint(4, 56), rng.randrange(1 << 20)
    if flow == "curv":
        n[0] = max(n[0], 44)  # both sponges, 20 cells each, within two blocks
    return {"use": use, "flow": flow, "nx": n[0], "ny": n[1], "nz": n[2], "precision": precision,
            "viscous": rng.choice([1, 1, 1, 0]), "steps": 10 if use == "host" else STEPS, "count": count,
            "layout": layout}


# ---------------------------------------------------------------------------
# inputs

def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def conserved(rho, u, v, w, p):
    q = [rho, rho * u, rho * v, rho * w, p / (GAM - 1) + 0.5 * rho * (u * u + v * v + w * w)]
    return torch.stack([t.expand(rho.shape) for t in q])


def to_host(t, pinned=False):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned and torch.cuda.is_available())
    out.copy_(t)
    return out.numpy()


def box_flow(r, nx, ny, nz, vortex=False, viscous=1):
    """One block periodic in every direction: a Taylor-Green vortex with a few
    random long waves, or an isentropic vortex, at a random Mach and Reynolds number."""
    mach, re = r.uniform(0.1, 0.5), r.uniform(400.0, 3200.0)
    f = dict(dtype=torch.float64, device=device())
    per = cases.BC_PERIODIC
    blk = cases.BlockSpec(nx, ny, nz, [[per, per]] * 3, [[0, 0]] * 3)
    length = 10.0 if vortex else 2 * math.pi
    x, y, z = (length * torch.arange(n + 1, **f) / n for n in (nx, ny, nz))
    if vortex:
        x, y = x - length / 2, y - length / 2
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    shape = blk.shape
    if vortex:
        eps, xc, yc = 5.0 * mach / (2 * math.pi), r.uniform(-1, 1), r.uniform(-1, 1)
        r2 = (X - xc) ** 2 + (Y - yc) ** 2
        du = eps * torch.exp(0.5 * (1 - r2))
        temp = 1.0 - 0.5 * (GAM - 1) * eps * eps * torch.exp(1 - r2)
        rho = (temp ** (1.0 / (GAM - 1))).expand(shape)
        u, v, w, p = mach - (Y - yc) * du, (X - xc) * du, torch.zeros((), **f), rho * temp / GAM
    else:
        u = mach * torch.sin(X) * torch.cos(Y) * torch.cos(Z)
        v = -mach * torch.cos(X) * torch.sin(Y) * torch.cos(Z)
        w = torch.zeros(shape, **f)
        for _ in range(3):
            k, ph, a = [r.randint(1, 3) for _ in range(3)], r.uniform(0, 2 * math.pi), 0.02 * mach
            u = u + a * torch.sin(k[0] * Y + ph)
            v = v + a * torch.sin(k[1] * Z + ph)
            w = w + a * torch.sin(k[2] * X + ph)
        p = 1.0 / GAM + mach * mach / 16.0 * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0)
        rho = GAM * p
    xyz = torch.stack([t.expand(shape) for t in (X, Y, Z)])
    return cases.CaseSpec([blk], viscous=viscous, reoo=re / mach, xyz=[to_host(xyz)],
                          qa=[to_host(conserved(rho, u, v, w, p), True)])


def flow_cases(case, seed):
    """The case list (one, or a batch) of a context, inputs from the seed."""
    r = random.Random(seed * 7919 + 17)
    nx, ny, nz, visc = case["nx"], case["ny"], case["nz"], case["viscous"]
    flow = case["flow"]
    if flow == "tgv":
        return [box_flow(r, nx, ny, nz, viscous=visc)]
    if flow == "batch":
        s = random.Random(case["layout"])
        return [box_flow(r, *(s.randint(32, 96) for _ in range(3)), vortex=i % 2 == 1, viscous=visc)
                for i in range(case["count"])]
    if flow == "curv":
        cs = cases.curvilinear_4block(nx, ny, nz, mach=r.uniform(0.3, 0.5), seed=seed, viscous=visc)
    elif flow == "vortex":  # uniform along z: one plane, repeated
        a = dict(mach=r.uniform(0.4, 0.6), strength=r.uniform(4, 6), xc=r.uniform(2, 4), viscous=visc)
        cs = cases.vortex(nx, ny, 12, **a)
        b = cs.blocks[0]
        b.lze = nz
        xyz, qa = (np.repeat(t[0][:, :1], nz + 1, axis=1) for t in (cs.xyz, cs.qa))
        xyz[2] = (16.0 / nx * np.arange(nz + 1))[:, None, None]
        cs.xyz, cs.qa = [xyz], [qa]
    else:
        cs = cases.reference_validation(nx, ny, nz) if flow == "validation" else cases.reference_toy(nx, ny, nz)
        shift = np.array([r.uniform(-0.1, 0.1), r.uniform(-0.1, 0.1), 0.0])[:, None, None, None]
        cs.qa = [cases.initialo(g + shift) for g in cs.xyz]
        cs.reoo *= r.uniform(0.5, 2.0)
        cs.viscous = visc
    cs.qa = [to_host(torch.from_numpy(q), True) for q in cs.qa]
    return [cs]


def field_input(case, seed):
    g = torch.Generator(device=device()).manual_seed(seed)
    shape = (case["nz"] + 1, case["ny"] + 1, case["nx"] + 1)
    f = torch.randn(shape, dtype=torch.float64, device=device(), generator=g)
    for d, n in enumerate(shape):  # noise over resolved waves
        i = torch.arange(n, dtype=torch.float64, device=device()).reshape([-1 if k == d else 1 for k in range(3)])
        f = f + sum(torch.sin(k * 2 * math.pi * i / (n - 1)) for k in range(1, 9))
    return to_host(f, True)


def prepare(case, seed):
    cl = flow_cases(case, seed)
    ctx = api.Context(cl, precision=PRECISION[case["precision"]], upload_state=False)
    blocks = [(c, b) for c, cs in enumerate(cl) for b in range(len(cs.blocks))]
    new = lambda shape: to_host(torch.zeros(shape, dtype=torch.float64), True)
    s = {"case": case, "ctx": ctx, "blocks": blocks, "cases": len(cl), "qa": [cl[c].qa[b] for c, b in blocks]}
    for cs in cl:
        cs.xyz = None  # the context has the grid
    if case["use"] == "operators":
        s["f"] = field_input(case, seed)
        s["out"] = [new(s["f"].shape) for _ in range(3)]
        return s
    n = [int(np.prod(q.shape)) for q in s["qa"]]
    s["flat"] = new(sum(n))  # one array per run, the blocks' states in turn
    at = np.cumsum([0] + n)
    s["out"] = [s["flat"][at[i]:at[i + 1]].reshape(q.shape) for i, q in enumerate(s["qa"])]
    return s


# ---------------------------------------------------------------------------
# one pass

def run(state):
    return {"run": run_steps, "record": run_record, "host": run_host,
            "operators": run_operators}[state["case"]["use"]](state)


def start_run(s):
    for c in range(s["cases"]):
        s["ctx"].set_time(np.zeros(6), c)
    for (c, b), q in zip(s["blocks"], s["qa"]):
        s["ctx"].set_state(b, q, c)


def read_state(s):
    for (c, b), out in zip(s["blocks"], s["out"]):
        s["ctx"].get_state_into(b, out, c)
    return s["flat"] if len(s["out"]) > 6 else list(s["out"])


def read_times(s):
    return np.stack([s["ctx"].time(c) for c in range(s["cases"])])


def run_steps(s):
    start_run(s)
    s["ctx"].step(s["case"]["steps"])
    return {"state": read_state(s), "time": read_times(s)}


def run_record(s):
    ctx = s["ctx"]
    start_run(s)
    ctx.record_enable(True)
    for _ in range(s["case"]["steps"]):
        ctx.step(1)
        ctx.record_accumulate()
        ctx.time()
    fields, times = [], []
    for c in range(s["cases"]):
        arrays, t = ctx.record_output(c)
        fields += arrays
        times.append(t)
    out = {"fields": fields if len(fields) <= 6 else np.concatenate([a.ravel() for a in fields]),
           "times": np.array(times, np.float32)}
    if s["case"]["precision"] != "mixed":
        out["state"] = read_state(s)
    return out


def run_host(s):
    for c in range(s["cases"]):
        s["ctx"].set_time(np.zeros(6), c)
    for q, out in zip(s["qa"], s["out"]):
        out[...] = q
    s["ctx"].step_host(s["case"]["steps"], s["out"], s["blocks"])
    return {"state": list(s["out"]), "time": read_times(s)}


def run_operators(s):
    """The calls of one derivative sweep and one filter pass of a host program."""
    ctx, f, out = s["ctx"], s["f"], s["out"]
    ctx.mpigo([f], 0, 1, 0, 1, 1)
    for nn in (1, 2, 3):
        ctx.deriv(0, f, out[nn - 1], nn, 1)
    g = f.copy()
    ctx.mpigo([g], 1, 1, 0, 1, 1)
    ctx.filte(0, g, 1, 1)
    return {"derivatives": list(out), "filtered": g}


def work(case):
    """Per point: every RK stage reads the state at its start and at the step's start,
    the 10 metric terms, and writes the new state; the filter reads and writes the state."""
    if case["flow"] == "batch":
        s = random.Random(case["layout"])
        pts = sum(math.prod(s.randint(32, 96) + 1 for _ in range(3)) for _ in range(case["count"]))
    else:
        pts = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1) * {"curv": 4, "toy": 6}.get(case["flow"], 1)
    if case["use"] == "operators":
        return {"bytes": 8 * pts * (1 + 3 + 1), "flops": pts * (3 * 14 + 22)}
    metric = 4 if case["precision"] == "mixed" else 8
    step = 4 * (15 * 8 + 10 * metric) + 80
    flops = 4 * (15 * 14 + (12 * 14 + 150 if case["viscous"] else 0) + 110) + 15 * 22
    extra = 80 + (120 * case["steps"] if case["use"] == "record" else 80 * case["steps"] if case["use"] == "host" else 0)
    return {"bytes": pts * (case["steps"] * step + extra), "flops": pts * case["steps"] * flops}


# ---------------------------------------------------------------------------
# the scheme in 64 bits

ALPHA, BETA, AA, AB = 4 / 9, 1 / 36, 20 / 27, 25 / 216
A0 = (-6.666666667794732, 9.000000000052879, 1.333333333178555, -0.0833333333455545)
L0 = (8.000000000449464, 6.000000000542)                # row 0: 1, alpha01, beta02
A1 = (-0.3506944444280639, 0.8249999999974599, 0.7444444444773477, 0.014583333334139971)
L1 = (0.09166666665902128, 1.3500000000438646, 0.2666666666794667)  # row 1: alpha10, 1, alpha12, beta13


class Operators:
    """Dense compact derivative and filter of a line, with its coupling to the neighbours."""

    def __init__(self, fltk, fltrbc):
        k = math.pi * fltk
        c1, c2, c3 = math.cos(k), math.cos(2 * k), math.cos(3 * k)
        f = 1 / (30 - 5 * c1 + 10 * c2 - 3 * c3)
        self.al, self.be = f * (-30 * c1 - 2 * c3), 0.5 * f * (18 + 9 * c1 + 6 * c2 - c3)
        self.fa = 30 * math.cos(0.5 * k) ** 4 * f
        self.fb, self.fc = -2 * self.fa / 5, self.fa / 15
        al, be, a, b, c, x = self.al, self.be, self.fa, self.fb, self.fc, fltrbc
        ln = math.log(x)
        n0 = 1 / (1 + al * x + be * x * x)
        e = (x - 1) * ((a + c) + (x + 1) * (b + x * c)) / ln
        f0 = [n0 * t for t in (a - 5 * e / 3, b + 10 * e / 21, c - 5 * e / 42, 5 * e / 252, -e / 630)]
        e = (x - 1) * (b + c * (x + 1)) / ln
        f1 = [a + b + c + 1627 * e / 1260, a + 10 * e / 21, b - 5 * e / 42, c + 5 * e / 252, -e / 630]
        e = c * (x - 1) / ln
        f2 = [b + c + 1627 * e / 1260, a - 5 * e / 3, a - 5 * e / 42, b + 5 * e / 252, c - e / 630]
        self.lhs = ({0: [[1, *L0], [L1[0], 1, *L1[1:]]], 1: [[1, ALPHA, BETA], [ALPHA, 1, ALPHA, BETA]]},
                    {0: [[1, al * n0, be * n0], [al + be * x, 1, al, be], [be, al, 1, al, be]],
                     1: [[1, al, be], [al, 1, al, be], [be, al, 1, al, be]]})
        row = lambda at, w, skip: [(-sum(w) if j == at else w[j - (j > at)]) for j in range(len(w) + 1)]
        self.rhs0 = ([row(0, A0, 0), row(1, A1, 1)], [row(0, f0, 0), row(1, f1, 1), row(2, f2, 2)])
        self.sums = [self.contraction(nt) for nt in (0, 1)]

    def system(self, n, nt, s0, s1):
        """A and B of a line of n points; an interface end leaves its first two rows of B empty."""
        lo, hi = (ALPHA, BETA) if nt == 0 else (self.al, self.be)
        a, b = np.zeros((n, n)), np.zeros((n, n))
        sten = [-AB, -AA, 0, AA, AB] if nt == 0 else \
            [self.fc, self.fb, self.fa, -2 * (self.fa + self.fb + self.fc), self.fa, self.fb, self.fc]
        h, m = len(sten) // 2, 2 + nt
        for i in range(n):
            for j, v in zip(range(i - 2, i + 3), (hi, lo, 1, lo, hi)):
                if 0 <= j < n:
                    a[i, j] = v
            if m <= i < n - m:
                b[i, i - h:i + h + 1] = sten
        sign = -1.0 if nt == 0 else 1.0
        for end, kind in ((0, s0), (1, s1)):
            for r, w in enumerate(self.lhs[nt][kind]):
                v = np.zeros(n)
                v[:len(w)] = w
                a[n - 1 - r if end else r] = v[::-1] if end else v
            rows = self.rhs0[nt] if kind == 0 else [[]] * m
            for r, w in enumerate(rows):
                v = np.zeros(n)
                v[:len(w)] = w
                if kind == 1 and nt == 1 and r == 2:  # the filter's third row keeps its stencil, less the neighbour's value
                    v[:6] = sten[1:]
                b[n - 1 - r if end else r] = sign * v[::-1] if end else v
        return a, b

    def contraction(self, nt):
        """Interface sums: weights of the own first 12 values and of the neighbour's."""
        n = 24
        a, b = self.system(n, nt, 0, 0)
        cut = a.copy()
        for i, j in ((11, 13), (12, 13), (12, 14)):
            cut[i - 1, j - 1] = 0
        for i, j in ((14, 12), (13, 12), (13, 11)):
            cut[i - 1, j - 1] = 0
        p = cut @ np.linalg.solve(a, b)
        return p[12:14, 12:], p[12:14, :12][:, ::-1]  # own, neighbour (nearest value first)

    def line(self, n, nt, s0, s1):
        """(D, G0, G1): out = D f + G0 f(side 0 neighbour) + G1 f(side 1 neighbour)."""
        a, b = self.system(n, nt, s0, s1)
        m = 2 + nt
        own, other = self.sums[nt]
        g = []
        for end, kind in ((0, s0), (1, s1)):
            c = np.zeros((n, 12))
            if kind == 1:
                sign = -1.0 if (nt == 0 and end) else 1.0
                for r in range(2):
                    i = n - 1 - r if end else r
                    b[i] = 0
                    if end:
                        b[i, n - 12:] = sign * own[r][::-1]
                    else:
                        b[i, :12] = own[r]
                    c[i] = sign * other[r]
                if nt == 1:
                    c[n - m if end else 2, 0] = self.fc
            g.append(c)
        d = np.linalg.solve(a, np.concatenate([b, g[0], g[1]], axis=1))
        if nt == 1:
            d[:, :n] += np.eye(n)
        return d[:, :n], d[:, n:n + 12], d[:, n + 12:]


def along(m, f, d):
    """m applied along direction d (0 xi, 1 eta, 2 zeta) of f (fields, z, y, x)."""
    if d == 0:
        return f @ m.T
    if d == 1:
        return m @ f
    return (m @ f.reshape(*f.shape[:-2], -1)).reshape(*f.shape[:-3], m.shape[0], *f.shape[-2:])


def interface(code):
    return code in (cases.BC_INTER_STRAIGHT, cases.BC_PERIODIC)


def gcbc(code):
    return code in (cases.BC_NON_REFLECTIVE, cases.BC_INTER_CURV)


class Exact:
    """One case advanced in 64 bits by torch."""

    def __init__(self, cs):
        self.cs, self.f = cs, dict(dtype=torch.float64, device=device())
        self.op = Operators(cs.fltk, cs.fltrbc)
        self.lines = {}
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), **self.f)
        self.nb = len(cs.blocks)
        for b, blk in enumerate(cs.blocks):
            for d in range(3):
                s = [1 if interface(c) else 0 for c in blk.nbc[d]]
                for nt in (0, 1):
                    self.lines[b, d, nt] = [t(m) for m in self.op.line(blk.shape[2 - d], nt, *s)]
        self.q = [t(q) for q in cs.qa]
        am = math.sqrt(sum(float(v) ** 2 for v in cs.amach))
        re = cs.reoo / am if am > 1e-8 else cs.reoo
        self.s0 = 111 / cs.tempoo
        self.s1 = (self.s0 + 1) / re
        self.umf = [float(v) for v in cs.amach]
        self.metrics([t(x) for x in cs.xyz])
        self.boundaries()
        self.sponge([t(x) for x in cs.xyz])
        self.n = self.ndt = 0
        self.dt = self.dts = self.dte = self.time = 0.0

    # -- lines
    def neighbour(self, fs, b, d, side, jump=None):
        """The neighbour's 12 values next to the face, nearest first."""
        blk = self.cs.blocks[b]
        src = fs[blk.mbcd[d][side]]
        n = src.shape[-1 - d]
        i = torch.arange(1, 13, device=device())
        v = src.index_select(src.dim() - 1 - d, i if side == 1 else n - 1 - i)
        if jump and blk.nbc[d][side] == cases.BC_PERIODIC:  # coordinates jump by the period
            face = lambda x, at: x.narrow(x.dim() - 1 - d, at, 1)
            v = v - face(src, 0 if side == 1 else n - 1) + face(fs[b], fs[b].shape[-1 - d] - 1 if side else 0)
        return v

    def apply(self, fs, d, nt, jump=False):
        out = []
        for b, blk in enumerate(self.cs.blocks):
            m, g0, g1 = self.lines[b, d, nt]
            r = along(m, fs[b], d)
            for side, g in ((0, g0), (1, g1)):
                if interface(blk.nbc[d][side]):
                    r += along(g, self.neighbour(fs, b, d, side, jump), d)
            out.append(r)
        return out

    def filter(self, fs):
        for d in (1, 2, 0):
            fs = self.apply(fs, d, 1)
        return fs

    # -- set-up
    def metrics(self, xyz):
        g = [self.apply(xyz, d, 0, True) for d in range(3)]
        co = []
        for b in range(self.nb):
            j = [[g[d][b][m] for d in range(3)] for m in range(3)]  # j[m][d] = d x_m / d xi_d
            co.append(torch.stack([torch.stack([
                j[(c + 1) % 3][(d + 1) % 3] * j[(c + 2) % 3][(d + 2) % 3]
                - j[(c + 2) % 3][(d + 1) % 3] * j[(c + 1) % 3][(d + 2) % 3] for c in range(3)]) for d in range(3)]))
        flat = self.filter([m.reshape(9, *m.shape[2:]) for m in co])
        self.met = [m.reshape(3, 3, *m.shape[1:]) for m in flat]  # [direction][component]
        self.yaco = [3.0 / sum(g[d][b][m] * self.met[b][d, m] for m in range(3) for d in range(3))
                     for b in range(self.nb)]

    def boundaries(self):
        a = np.array([[L0[0], L0[1], 0, 0], [1, L1[1], L1[2], 0], [ALPHA, 1, ALPHA, BETA], [BETA, ALPHA, 1, ALPHA]])
        w = -np.linalg.solve(a, [1, L1[0], BETA, 0])
        w = [1.0] + [0.5 * w[i] * (1 + math.cos((i + 1) * math.pi / 5)) for i in range(4)]
        self.faces = []
        count = [torch.zeros_like(y) for y in self.yaco]
        for b, blk in enumerate(self.cs.blocks):
            for d in range(3):
                for side in range(2):
                    if gcbc(blk.nbc[d][side]):
                        n = count[b].shape[2 - d]
                        for i in range(5):
                            count[b].select(2 - d, n - 1 - i if side else i).add_(1)
        for b, blk in enumerate(self.cs.blocks):
            for d in range(3):
                for side in range(2):
                    if not gcbc(blk.nbc[d][side]):
                        continue
                    n = count[b].shape[2 - d]
                    at = [n - 1 - i if side else i for i in range(5)]
                    ya = self.yaco[b].select(2 - d, at[0])
                    m = self.met[b][d].select(3 - d, at[0]) * ya
                    self.faces.append({"b": b, "d": d, "side": side, "at": at, "code": blk.nbc[d][side], "yaco": ya,
                                       "cm": m / m.square().sum(0).sqrt(),
                                       "w": [w[i] / ya / count[b].select(2 - d, at[i]) for i in range(5)]})

    def sponge(self, xyz):
        cs, self.sp = self.cs, None
        if cs.szco == 0.0:
            return
        self.sp = []
        for b, x in enumerate(xyz):
            c = [torch.cos((math.pi / w * v).clamp(0, math.pi)) for w, v in (
                (cs.szth0, x[0] + cs.doml0 - cs.szth0), (cs.szth1, cs.doml1 - cs.szth1 - x[0]))]
            a, m = 0.5 * cs.szco * (2 + c[0] + c[1]), 0.5 * cs.szco * (1 + c[0])
            on = (a > 1e-8).double()
            self.sp.append((on * a / self.yaco[b], on * m / self.yaco[b]))

    # -- one step
    def primitives(self, b):
        q = self.q[b]
        rho = 1 / q[0]
        u = q[1:4] * rho
        p = (GAM - 1) * (q[4] - 0.5 * (q[1:4] * u).sum(0))
        return rho, u, p, GAM * p * rho

    def time_step(self):
        if self.n % 10 == 1:
            self.ndt, self.dts, r = self.n, self.dte, [0.0, 0.0]
            for b in range(self.nb):
                rho, u, p, temp = self.primitives(b)
                m, ya = self.met[b], self.yaco[b].abs()
                m2 = m.square().sum((0, 1))
                un = sum(sum(m[d, c] * (u[c] + self.umf[c]) for c in range(3)).abs() for d in range(3))
                mu = self.s1 * temp ** 1.5 / (temp + self.s0)
                r = [max(r[0], float((((temp * m2).sqrt() + un) * ya).max())),
                     max(r[1], float((rho * mu * m2 * ya * ya).max()))]
            self.dte = self.cs.cfl / r[0]
            if self.cs.viscous:
                self.dte = min(self.dte, 0.5 / r[1])
        self.dt = self.dts + (self.dte - self.dts) * math.sin(0.05 * math.pi * (self.n - self.ndt)) ** 2

    def rhs(self):
        prim = [self.primitives(b) for b in range(self.nb)]
        if self.cs.viscous:
            g = [self.apply([torch.cat([pr[1], pr[3][None]]) for pr in prim], d, 0) for d in range(3)]
        flux = []
        for b in range(self.nb):
            rho, u, p, temp = prim[b]
            q, m = self.q[b], self.met[b]
            ut = [u[c] + self.umf[c] for c in range(3)]
            tau = heat = None
            if self.cs.viscous:
                mu = self.yaco[b] * self.s1 * temp ** 1.5 / (temp + self.s0)
                grad = [[sum(m[d, c] * g[d][b][i] for d in range(3)) for c in range(3)] for i in range(4)]
                div = (grad[0][0] + grad[1][1] + grad[2][2]) * (2.0 / 3.0)
                tau = [[mu * (grad[i][j] + grad[j][i] - (div if i == j else 0)) for j in range(3)] for i in range(3)]
                heat = [mu * grad[3][j] / ((GAM - 1) * PRNDTL) + sum(u[i] * tau[i][j] for i in range(3)) for j in range(3)]
            block = []
            for d in range(3):
                un = sum(m[d, c] * ut[c] for c in range(3))
                f = torch.empty_like(q)
                f[0] = q[0] * un
                for c in range(3):
                    f[c + 1] = q[c + 1] * un + m[d, c] * p
                f[4] = (q[4] + p) * un - p * sum(self.umf[c] * m[d, c] for c in range(3))
                if tau:
                    for c in range(3):
                        f[c + 1] -= sum(m[d, j] * tau[c][j] for j in range(3))
                    f[4] -= sum(m[d, j] * heat[j] for j in range(3))
                block.append(f)
            flux.append(block)
        de, ends = [0.0] * self.nb, {}
        for d in range(3):
            r = self.apply([flux[b][d] for b in range(self.nb)], d, 0)
            for face in self.faces:
                if face["d"] == d:
                    ends[id(face)] = r[face["b"]].select(3 - d, face["at"][0]).clone()
            de = [de[b] + r[b] for b in range(self.nb)]
        self.characteristic(de, ends, prim)
        if self.sp:
            for b, (a, m) in enumerate(self.sp):
                q, rest = self.q[b], 1 / (GAM * (GAM - 1))
                de[b] += torch.stack([a * (q[0] - 1), m * q[1], m * q[2], m * q[3], a * (q[4] - rest)])
        return de

    def characteristic(self, de, ends, prim):
        """The non-reflecting and the curved-interface faces (waves normal to the face)."""
        if not self.faces:
            return
        at = lambda t, f: t.select(t.dim() - 1 - f["d"], f["at"][0])
        for f in self.faces:
            b, cm = f["b"], f["cm"]
            rho, u, p, temp = prim[b]
            u, ao = at(u, f), at(temp, f).sqrt()
            hv, vn = 0.5 * u.square().sum(0), (cm * u).sum(0)
            vs = sum(cm[c] * self.umf[c] for c in range(3))
            ho = (GAM - 1) / ao ** 2
            v = f["yaco"] * (ends[id(f)] if f["code"] == cases.BC_NON_REFLECTIVE else at(de[b], f))
            # entropy/vorticity and the two acoustic waves of the change v
            dp = ho * (hv * v[0] - (u * v[1:4]).sum(0) + v[4])       # dp / ao^2
            du = (v[1:4] - u * v[0]) / ao                            # rho du / ao
            cross = torch.stack([cm[1] * du[2] - cm[2] * du[1], cm[2] * du[0] - cm[0] * du[2], cm[0] * du[1] - cm[1] * du[0]])
            dn = (cm * du).sum(0)
            wave = torch.cat([cm * (v[0] - dp) - cross, (dp + dn)[None], (dp - dn)[None]])
            f.update(wave=wave, u=u, ao=ao, hv=hv, vn=vn, vs=vs)
        by = {(f["b"], f["d"], f["side"]): f for f in self.faces}
        for f in self.faces:
            b, d, cm, u, ao = f["b"], f["d"], f["cm"], f["u"], f["ao"]
            s, un = 1 - 2 * f["side"], f["vn"] + f["vs"]
            new = f["wave"].clone()
            if f["code"] == cases.BC_NON_REFLECTIVE:
                new[3] = torch.where(s * (un + ao) > 0, 0.0, new[3])
                new[4] = torch.where(s * (un - ao) > 0, 0.0, new[4])
            else:
                o = by[self.cs.blocks[b].mbcd[d][f["side"]], d, 1 - f["side"]]["wave"]
                new[:3] = torch.where(s * un > 0, o[:3], new[:3])
                new[3] = torch.where(s * (un + ao) > 0, o[3], new[3])
                new[4] = torch.where(s * (un - ao) > 0, o[4], new[4])
            w = new - f["wave"]
            ent, dp, dn = (cm * w[:3]).sum(0), 0.5 * (w[3] + w[4]), 0.5 * (w[3] - w[4])
            mom = ao * (torch.stack([cm[1] * w[2] - cm[2] * w[1], cm[2] * w[0] - cm[0] * w[2], cm[0] * w[1] - cm[1] * w[0]])
                        + cm * dn)
            drho = ent + dp
            dm = mom + u * drho
            r = torch.cat([drho[None], dm, (f["hv"] * drho + (u * mom).sum(0) + ao ** 2 / (GAM - 1) * dp)[None]])
            for i in range(5):
                de[b].select(3 - d, f["at"][i]).add_(f["w"][i] * r)

    def average(self):
        """Points stored more than once: on block edges the mean over the blocks that meet
        there, then face by face the running mean with the copy across the face (in the
        order xi, eta, zeta, so an edge of a block that is periodic onto itself weighs the
        copies across its two faces and not the one across both)."""
        linked = lambda blk, d, side: blk.nbc[d][side] in (
            cases.BC_INTER_STRAIGHT, cases.BC_PERIODIC, cases.BC_INTER_CURV)
        cut = lambda t, d, side: t.select(t.dim() - 1 - d, t.shape[t.dim() - 1 - d] - 1 if side else 0)
        for d in range(3):
            new = []
            for b, blk in enumerate(self.cs.blocks):
                edge = torch.zeros(blk.shape, dtype=torch.bool, device=device())
                for e in range(3):
                    for side in range(2):
                        if e != d and blk.mbcd[e][side] >= 0:
                            cut(edge, e, side).fill_(True)
                for side in range(2):
                    if linked(blk, d, side) and blk.mbcd[d][side] != b:
                        q, o = cut(self.q[b], d, side), cut(self.q[blk.mbcd[d][side]], d, 1 - side)
                        new.append((q, torch.where(cut(edge, d, side), 0.5 * (q + o), q)))
            for q, v in new:
                q.copy_(v)
        old = [{(d, side): cut(q, d, side).clone() for d in range(3) for side in range(2)} for q in self.q]
        for b, blk in enumerate(self.cs.blocks):
            r = torch.ones(blk.shape, **self.f)
            for d in range(3):
                for side in range(2):
                    if linked(blk, d, side):
                        n, q = cut(r, d, side), cut(self.q[b], d, side)
                        n.add_(1)
                        q.copy_(((n - 1) * q + old[blk.mbcd[d][side]][d, 1 - side]) / n)

    def step(self):
        self.q = self.filter(self.q)
        start = [q.clone() for q in self.q]
        self.time_step()
        for nk in range(1, 5):
            de = self.rhs()
            self.q = [start[b] - self.dt / (5 - nk) * self.yaco[b] * de[b] for b in range(self.nb)]
            self.average()
        self.start = start
        self.n += 1
        self.time += self.dt


def exact(case, seed):
    cl = flow_cases(case, seed)
    host = lambda t: t.cpu().numpy()
    if case["use"] == "operators":
        e = Exact(cl[0])
        f = torch.as_tensor(field_input(case, seed), **e.f)
        return {"derivatives": [host(e.apply([f[None]], d, 0)[0][0]) for d in range(3)],
                "filtered": host(e.apply([f[None]], 1, 1)[0][0])}
    state, times, fields, mid = [], [], [], []
    for cs in cl:
        e = Exact(cs)
        record = case["use"] == "record"
        mean, span = [0.0] * e.nb, 0.0
        for _ in range(case["steps"]):
            e.step()
            if record:
                mean = [mean[b] + 0.5 * e.dt * (e.start[b] + e.q[b]) for b in range(e.nb)]
                span += e.dt
        state += [host(q) for q in e.q]
        times.append([e.n, e.ndt, e.dt, e.dts, e.dte, e.time])
        if record:
            mid.append(e.time - 0.5 * span)
            for b in range(e.nb):
                q = mean[b] / span
                u = q[1:4] / q[0]
                p = (GAM - 1) * (q[4] - 0.5 * (q[1:4] * u).sum(0))
                um = torch.tensor(e.umf, **e.f)[:, None, None, None]
                fields.append(host(torch.cat([q[:1], u + um, p[None]])))
    flat = lambda v: v if len(v) <= 6 else np.concatenate([a.ravel() for a in v])
    if case["use"] == "record":
        out = {"fields": flat(fields), "times": np.array(mid)}
        if case["precision"] != "mixed":
            out["state"] = flat(state)
        return out
    return {"state": flat(state), "time": np.array(times)}
