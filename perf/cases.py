"""Timed workloads of the MPDATA and Boussinesq solvers: the calls a program makes, over the sizes it makes them at.

A pass is what a time loop does between two looks at the fields: advance(nt) on a run object (or a
batch of them) whose fields live on the device, then every advected field fetched into the program's
own device tensors.  The state goes on from pass to pass, as it does in such a loop.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  run object, loaded fields, output tensors
    run(state)           one pass
    work(case)           bytes and operations that one pass cannot do without
    exact(case, seed)    the first pass in 64-bit torch, from the formulae alone

Case keys: solver (mpdata, batch, boussinesq), grid, bc (cyclic, open), flow (uniform, rotation, curl),
opts, n_iters, dtype, n_eqns, nt (steps per pass); batch: problems, lo, hi, sizes_seed; boussinesq:
prs_k (1: cr, more: gcrk), prs_fp64, iters (about how many GCR iterations a solve of this size takes).
"""
import functools
import math
import random

import torch

from libmpdataxx_b200 import _lib, bcond, concurr, opts, solvers

DEV = "cuda" if torch.cuda.is_available() else "cpu"
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    adv = {"solver": "mpdata", "n_eqns": 1}
    return [
        # the smallest problem: a 1D box, many steps per call; latency of one step
        dict(adv, name="box_1d_2000", grid="2000", bc="cyclic", flow="uniform", opts="0", n_iters=2, dtype="f64", nt=100),
        # two advected quantities of one 1D flow with the limiter (option comparison of the advection schemes)
        dict(adv, name="options_1d_601", grid="601", bc="cyclic", flow="uniform", opts="iga|fct", n_iters=2, dtype="f64",
             n_eqns=2, nt=20),
        # the rotating cone, open boundaries: an ordinary small 2D run
        dict(adv, name="cone_2d_101_open", grid="101x101", bc="open", flow="rotation", opts="iga|fct", n_iters=2,
             dtype="f64", nt=10),
        # 2D rotation with FCT and three iterations at the size the 2D figures are quoted on
        dict(adv, name="rotation_2d_1024", grid="1024x1024", bc="cyclic", flow="rotation", opts="fct", n_iters=3,
             dtype="f64", nt=10),
        # the revolving sphere, open boundaries: an ordinary small 3D run
        dict(adv, name="sphere_3d_59_open", grid="59x59x59", bc="open", flow="rotation", opts="fct", n_iters=2, dtype="f64",
             nt=5),
        # third-order terms, infinite gauge and FCT on a larger ragged open domain in single precision
        dict(adv, name="sphere_3d_ragged_open", grid="163x150x177", bc="open", flow="rotation", opts="iga|tot|fct",
             n_iters=2, dtype="f32", nt=3),
        # the headline: one big periodic deformational flow in single precision
        dict(adv, name="flow_3d_512", grid="512x512x512", bc="cyclic", flow="curl", opts="iga|fct", n_iters=2, dtype="f32",
             nt=4),
        # the same in double precision (the default type) on an odd-sized grid
        dict(adv, name="flow_3d_ragged_f64", grid="250x257x241", bc="cyclic", flow="curl", opts="iga|fct", n_iters=2,
             dtype="f64", nt=4),
        # an ensemble of independent 2D problems of uneven sizes
        {"name": "ensemble_2d_256", "solver": "batch", "problems": 256, "lo": 64, "hi": 1024, "sizes_seed": 5,
         "flow": "curl", "opts": "fct", "n_iters": 2, "dtype": "f32", "n_eqns": 1, "bc": "cyclic", "nt": 4},
        # the 2D buoyant thermal
        {"name": "thermal_2d_201", "solver": "boussinesq", "grid": "201x201", "bc": "cyclic", "opts": "iga|fct",
         "n_iters": 2, "dtype": "f64", "prs_k": 1, "prs_fp64": False, "nt": 2, "iters": 60},
        # a small ragged 3D bubble between walls with the longer GCR basis
        {"name": "bubble_3d_gcrk", "solver": "boussinesq", "grid": "97x89x65", "bc": "walls", "opts": "iga|fct",
         "n_iters": 2, "dtype": "f64", "prs_k": 3, "prs_fp64": False, "nt": 1, "iters": 12},
        # the large 3D bubble: single-precision advection, double-precision pressure solve
        {"name": "bubble_3d_256", "solver": "boussinesq", "grid": "256x256x128", "bc": "walls", "opts": "iga|fct",
         "n_iters": 2, "dtype": "f32", "prs_k": 1, "prs_fp64": True, "nt": 1, "iters": 70},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["1d", "2d", "2d", "3d", "3d", "batch", "thermal", "bubble"])
    dtype = rng.choice(["f32", "f64"])
    if kind == "batch":
        lo = log(32, 256)
        return {"solver": "batch", "problems": log(4, 128), "lo": lo, "hi": lo + log(16, 512), "sizes_seed": rng.randrange(10 ** 6),
                "flow": "curl", "opts": rng.choice(["fct", "iga|fct", "0"]), "n_iters": 2, "dtype": dtype, "n_eqns": 1,
                "bc": "cyclic", "nt": rng.randint(2, 6)}
    if kind in ("thermal", "bubble"):
        g = [log(48, 400), log(48, 400)] if kind == "thermal" else [log(24, 160), log(24, 160), log(20, 96)]
        return {"solver": "boussinesq", "grid": "x".join(map(str, g)), "bc": "cyclic" if kind == "thermal" else "walls",
                "opts": "iga|fct", "n_iters": 2, "dtype": dtype, "prs_k": rng.choice([1, 1, 2, 3, 4]),
                "prs_fp64": dtype == "f32", "nt": rng.randint(1, 2), "iters": 50 if kind == "thermal" else 30}
    nd = int(kind[0])
    g = {1: lambda: [log(64, 20000)], 2: lambda: [log(32, 1500) for _ in range(2)],
         3: lambda: [log(20, 260) for _ in range(3)]}[nd]()
    bc = rng.choice(["cyclic", "cyclic", "open"])
    o = rng.choice(["0", "fct", "iga|fct", "iga|fct", "iga", "iga|tot|fct", "tot|fct"])
    return {"solver": "mpdata", "n_eqns": rng.choice([1, 1, 1, 2]), "grid": "x".join(map(str, g)), "bc": bc,
            "flow": "uniform" if nd == 1 else ("rotation" if bc == "open" else "curl"), "opts": o,
            "n_iters": 3 if "iga" not in o and rng.random() < 0.4 else 2, "dtype": dtype,
            "nt": {1: 40, 2: 8, 3: 3}[nd] + rng.randint(0, 3)}


# ---------------------------------------------------------------------------
# inputs

def _bits(case):
    b = 0
    for w in case["opts"].split("|"):
        b |= 0 if w == "0" else getattr(opts, w)
    return b


def _grid(case):
    return tuple(int(g) for g in case["grid"].split("x"))


def _axes(sizes):
    """Index vectors 0..n-1 of each axis, shaped to broadcast against each other."""
    nd = len(sizes)
    return [torch.arange(n, dtype=torch.float64, device=DEV).reshape([-1 if q == d else 1 for q in range(nd)])
            for d, n in enumerate(sizes)]


def _modes(P, rng, m=8):
    """Sum of m random Fourier modes on the periodic box of P points per axis (wave numbers 1..4)."""
    ang = lambda n, k: (2 * math.pi / n) * torch.outer(torch.tensor([float(q) for q in k], dtype=torch.float64, device=DEV),
                                                      torch.arange(n, dtype=torch.float64, device=DEV))
    ks = [[rng.randint(1, 4) for _ in range(m)] for _ in P]
    amp = torch.tensor([rng.gauss(0, 1) for _ in range(m)], dtype=torch.float64, device=DEV)
    ph = torch.tensor([rng.uniform(0, 2 * math.pi) for _ in range(m)], dtype=torch.float64, device=DEV)
    u = ang(P[0], ks[0]) + ph[:, None]
    for d in range(1, len(P) - 1):
        u = (u[:, :, None] + ang(P[d], ks[d])[:, None, :]).reshape(m, -1)
    v = ang(P[-1], ks[-1])
    return (torch.cos(u).t() @ (amp[:, None] * torch.cos(v)) - torch.sin(u).t() @ (amp[:, None] * torch.sin(v))).reshape(P)


def _wrap(x, n, d, first):
    """Points first, first + 1, ... of the periodic array x along axis d, n of them."""
    return x.index_select(d, (torch.arange(n, device=DEV) + first) % x.shape[d])


def _views(faces, grid):
    """Advector views (lower bound -1 along x; along the own axis too) of unique periodic faces."""
    out = []
    for d, f in enumerate(faces):
        for q, n in enumerate(grid):
            f = _wrap(f, n + 1 if q == 0 and d > 0 else n, q, -1 if q == 0 or q == d else 0)
        out.append(f.contiguous())
    return out


def _curl(grid, rng, cmax, dt):
    P = tuple(n - 1 for n in grid)
    back = lambda x, d: torch.roll(x, 1, d)
    if len(grid) == 2:
        s = _modes(P, rng)
        f = [s - back(s, 1), back(s, 0) - s]
    else:
        a = [_modes(P, rng) for _ in range(3)]
        f = [(a[2] - back(a[2], 1)) - (a[1] - back(a[1], 2)), (a[0] - back(a[0], 2)) - (a[2] - back(a[2], 0)),
             (a[1] - back(a[1], 0)) - (a[0] - back(a[0], 1))]
        del a
    s = cmax / max(float(x.abs().max()) for x in f)
    return _views([(x * s).to(dt) for x in f], grid)


def _rotation(case, grid, dt):
    """Solid-body rotation about the centre: each component is constant along its own axis."""
    nd, cyc = len(grid), case["bc"] == "cyclic"
    out = []
    for d in range(nd):
        size = [n + (1 if q == 0 and d > 0 else 0) for q, n in enumerate(grid)]
        x = []
        for q, a in enumerate(_axes(size)):
            a = a - 1 if q == 0 or q == d else a
            P = grid[q] - 1
            x.append(torch.clamp((a % P if cyc else a) / P - 0.5, -0.48, 0.48) if cyc else a / P - 0.5)
        if nd == 2:
            f = x[1] if d == 0 else -x[0]
        else:
            f = (x[2] - x[1], x[0] - x[2], x[1] - x[0])[d]
        out.append(((0.9 if nd == 2 else 0.35) * f).expand(size).to(dt).contiguous())
    return out


def _blob(case, grid, rng):
    """A cone (2D) or ball (3D) off the centre, or Gaussian blobs where the flow is deformational."""
    nd, P = len(grid), [n - 1 for n in grid]
    if case["flow"] == "curl":
        if case["solver"] == "batch":
            g = torch.Generator(device=DEV)
            g.manual_seed(rng.randrange(1 << 40))
            u = torch.randn(P, generator=g, device=DEV, dtype=torch.float64).exp()
        else:
            u = torch.zeros(P, dtype=torch.float64, device=DEV)
            for _ in range(5):
                e = []
                for q, a in enumerate(_axes(P)):
                    d = (a - rng.uniform(0, P[q])).abs()
                    d = torch.minimum(d, P[q] - d) / (0.05 * P[q])
                    e.append(torch.exp(-0.5 * d * d))
                u += functools.reduce(torch.mul, e)
        for q, n in enumerate(grid):
            u = _wrap(u, n, q, 0)
        return u
    ax = [a / p for a, p in zip(_axes(grid), P)]
    if case["bc"] == "cyclic":
        ax = [a % 1.0 for a in ax]
    th, h = rng.uniform(0, 2 * math.pi), rng.uniform(3, 5)
    c = [0.5 + 0.25 * math.cos(th), 0.5 + 0.25 * math.sin(th), 0.5 + rng.uniform(-0.1, 0.1)][:nd]
    r = torch.sqrt(sum((a - q) ** 2 for a, q in zip(ax, c))) / 0.15
    if nd == 2:
        return (1.0 if case["bc"] == "open" else 0.0) + torch.clamp(h * (1 - r), min=0)
    return torch.where(r <= 1, h, 0.0)


def _fields(case, grid, rng):
    """([advectee per equation], [advector per axis]) of one mpdata problem."""
    dt = DTYPES[case["dtype"]]
    if len(grid) == 1:
        n, psi = grid[0], []
        for e in range(case["n_eqns"]):
            a = torch.tensor([0.1 + rng.uniform(0, 0.01) for _ in range(n)], dtype=torch.float64, device=DEV)
            lo = rng.randint(n // 10, n // 5)
            a[lo:lo + max(1, n // 10)] = 1.0 + e
            if case["bc"] == "cyclic":
                a[-1] = a[0]
            psi.append(a.to(dt))
        return psi, [torch.full((n,), 0.5, dtype=dt, device=DEV)]
    adv = _curl(grid, rng, 0.3, dt) if case["flow"] == "curl" else _rotation(case, grid, dt)
    return [_blob(case, grid, rng).to(dt).contiguous() for _ in range(case["n_eqns"])], adv


def _problems(case, seed):
    rng = random.Random(1000003 * int(seed) + 17)
    if case["solver"] != "batch":
        yield _grid(case), _fields(case, _grid(case), rng)
        return
    sizes = random.Random(case["sizes_seed"])
    for _ in range(case["problems"]):
        g = (sizes.randint(case["lo"], case["hi"]), sizes.randint(case["lo"], case["hi"]))
        yield g, _fields(case, g, rng)


def _thermal(case, seed):
    """Velocities at rest and a warm disc or ball (seeded place and noise) in the environment tht_e."""
    grid, rng = _grid(case), random.Random(1000003 * int(seed) + 29)
    nd, dt, dx = len(grid), DTYPES[case["dtype"]], 10.0
    ax = [a * dx for a in _axes(grid)]
    L = [(n - 1) * dx for n in grid]
    tht_e = (torch.full(grid, 300.0, dtype=torch.float64, device=DEV) if nd == 2
             else (300.0 * torch.exp(1e-4 * ax[-1] / 9.81)).expand(grid))
    c = [(0.5 + rng.uniform(-0.02, 0.02)) * l for l in L]
    c[-1] = (0.13 if nd == 2 else 0.25) * L[-1] + rng.uniform(0, 0.02) * L[-1]
    r = (0.125 if nd == 2 else 0.1) * L[0]
    inside = sum((a - q) ** 2 for a, q in zip(ax, c)) <= r * r
    tht = tht_e + torch.where(inside, 0.5, 0.0)
    if nd == 3:
        g = torch.Generator(device=DEV)
        g.manual_seed(rng.randrange(1 << 40))
        tht = tht + 0.02 * torch.rand(grid, generator=g, device=DEV, dtype=torch.float64) - 0.01
    for q in range(nd):  # the last point of a cyclic axis is its first
        if case["bc"] == "cyclic" or q < nd - 1:
            tht.select(q, grid[q] - 1).copy_(tht.select(q, 0))
    return [torch.zeros(grid, dtype=dt, device=DEV) for _ in range(nd)] + [tht.to(dt).contiguous()], tht_e.to(dt).contiguous()


# ---------------------------------------------------------------------------
# the calls

def _ct(case, nd, n_eqns):
    class ct(solvers.ct_params_default_t):
        pass
    ct.real_t = {"f32": "float32", "f64": "float64"}[case["dtype"]]
    ct.n_dims, ct.n_eqns, ct.opts = nd, n_eqns, _bits(case)
    return ct


def _mpdata(case, grid, psi, adv):
    p = solvers.mpdata.rt_params_t(grid_size=list(grid), n_iters=case["n_iters"], max_abs_div_eps=1e-5)
    r = concurr.cuda(solvers.mpdata(_ct(case, len(grid), len(psi))), *[getattr(bcond, case["bc"])] * (2 * len(grid)), p=p)
    _load(r, psi, adv)
    return r


def _load(r, psi, adv=()):
    for e, a in enumerate(psi):
        r.set_field_device(_lib.FIELD_ADVECTEE, e, a.data_ptr())
    for d, a in enumerate(adv):
        r.set_field_device(_lib.FIELD_ADVECTOR, d, a.data_ptr())


def prepare(case, seed):
    if case["solver"] == "boussinesq":
        grid = _grid(case)
        nd = len(grid)
        psi, tht_e = _thermal(case, seed)
        ct = _ct(case, nd, nd + 1)
        ct.rhs_scheme = solvers.trapez
        ct.prs_scheme = solvers.cr if case["prs_k"] == 1 else solvers.gcrk
        ct.prs_k_iters = case["prs_k"]

        class ix:
            vip_i, vip_j, vip_k, tht = 0, 1, 2, nd
        ct.ix = ix
        p = solvers.boussinesq.rt_params_t(grid_size=list(grid), n_iters=case["n_iters"], dt=0.75, di=10.0, dj=10.0, dk=10.0,
                                           prs_tol=1e-7, g=9.81, Tht_ref=300.0, prs_fp64=case["prs_fp64"])
        bcs = [bcond.cyclic] * (2 * nd) if case["bc"] == "cyclic" else [bcond.cyclic] * (2 * nd - 2) + [bcond.rigid] * 2
        r = concurr.cuda(solvers.boussinesq(ct), *bcs, p=p)
        r.set_field_device(_lib.FIELD_SCLR_ARRAY, _lib.SCLR_THT_E, tht_e.data_ptr())
        _load(r, psi)
        return {"case": case, "step": r, "runs": [r], "out": [[torch.empty_like(a) for a in psi]]}
    runs, out = [], []
    for grid, (psi, adv) in _problems(case, seed):
        runs.append(_mpdata(case, grid, psi, adv))
        out.append([torch.empty_like(a) for a in psi])
    return {"case": case, "step": concurr.batch(runs) if case["solver"] == "batch" else runs[0], "runs": runs, "out": out}


def run(state):
    state["step"].advance(state["case"]["nt"])
    if state["case"]["solver"] == "batch":
        state["step"].sync()
    for r, fields in zip(state["runs"], state["out"]):
        for e, a in enumerate(fields):
            r.get_field_device(_lib.FIELD_ADVECTEE, e, a.data_ptr())
    return state["out"] if len(state["runs"]) <= 32 else torch.cat([a.reshape(-1) for f in state["out"] for a in f])


def work(case):
    """Advection: per step and equation psi in and out, per step the advector; then the fetched fields read and
    written.  GCR: per iteration and direction the fields that the recurrences read and write.  What fits on the chip
    (64 MB) counts once per pass.  Operations: additions, multiplications, comparisons and divisions of the formulae
    per point and step, counted once per face."""
    chip = 2 ** 26
    es = 4 if case["dtype"] == "f32" else 8
    if case["solver"] == "batch":
        sizes = random.Random(case["sizes_seed"])
        cells = sum(sizes.randint(case["lo"], case["hi"]) * sizes.randint(case["lo"], case["hi"]) for _ in range(case["problems"]))
        nd, ne = 2, 1
    else:
        nd, cells = len(_grid(case)), math.prod(_grid(case))
        ne = nd + 1 if case["solver"] == "boussinesq" else case["n_eqns"]
    ops = {1: 20, 2: 60, 3: 130}[nd] * (case["n_iters"] - 1) * (2 if "fct" in case["opts"] else 1)
    one = cells * es * (2 * ne + nd)
    byt = (case["nt"] if one > chip else 1) * one + 2 * ne * cells * es
    flo = case["nt"] * cells * ne * ops
    if case["solver"] == "boussinesq":
        ps = 8 if case["prs_fp64"] else es
        k = case["prs_k"]
        per = sum(10 + 2 * v for v in range(1, k + 1))  # inner step v: err, lap_err, Phi, v directions and their laps
        one = cells * (per * ps + (6 * nd + 6) * es)
        byt += case["nt"] * (case["iters"] * cells * per * ps + cells * (6 * nd + 6) * es) if one > chip else one
        flo += case["nt"] * cells * case["iters"] * k * (40 + 6 * k)
    return {"bytes": float(byt), "flops": float(flo)}


# ---------------------------------------------------------------------------
# the first pass in 64 bits, from the formulae of the scheme (arrays with a halo of 2 on every side)

H = 2


class _mp:
    def __init__(self, case, grid, psi, adv):
        self.o, self.n, self.nd, self.bc, self.ni = set(case["opts"].split("|")), grid, len(grid), case["bc"], case["n_iters"]
        i = torch.finfo(DTYPES[case["dtype"]])
        self.tiny, self.eps = i.tiny, i.eps
        shape = [n + 2 * H for n in grid]
        z = lambda: torch.zeros(shape, dtype=torch.float64, device=DEV)
        self.p, self.g = z(), []
        self.p[tuple(slice(H, H + n) for n in grid)] = psi.double()
        for d, a in enumerate(adv):
            g = z()
            lo = [H - (1 if q == 0 or q == d else 0) for q in range(self.nd)]
            g[tuple(slice(l, l + m) for l, m in zip(lo, a.shape))] = a.double()
            self.g.append(g)
        self.along(self.g, False)
        for d in range(self.nd):
            self.normal(self.g, d)

    def at(self, d, *idx, others=None):
        """Index of planes idx (or a range) along axis d; the other axes whole, or as `others` says."""
        s = [slice(None)] * self.nd
        for q, v in (others or {}).items():
            s[q] = v
        s[d] = slice(idx[0] + H, idx[1] + H) if len(idx) == 2 else idx[0] + H
        return tuple(s)

    def scalar(self, a, axes=None):
        for d in range(self.nd) if axes is None else axes:
            n = self.n[d]
            if self.bc == "cyclic":
                a[self.at(d, -H, 0)] = a[self.at(d, n - 1 - H, n - 1)].clone()
                a[self.at(d, n, n + H)] = a[self.at(d, 1, 1 + H)].clone()
            else:
                a[self.at(d, -H, 0)] = a[self.at(d, 0, 1)]
                a[self.at(d, n, n + H)] = a[self.at(d, n - 1, n)]

    def along(self, v, ad):
        k = 1 if ad else 0
        for d in range(self.nd):
            a, n = v[d], self.n[d]
            if self.bc == "cyclic":
                a[self.at(d, -H, 0)] = a[self.at(d, n - 1 - H, n - 1)].clone()
                a[self.at(d, n - 1, n - 1 + H)] = a[self.at(d, 0, H)].clone()
                continue
            if self.nd == 1:
                a[self.at(0, -H, -k)] = a[self.at(0, 0, 1)].clone()
                a[self.at(0, n - 1 + k, n - 1 + H)] = a[self.at(0, n - 1 - H, n - H)].clone()
                continue
            core = {q: slice(H, H + self.n[q]) for q in range(self.nd) if q != d}
            for side in (0, 1):  # zero divergence in the outermost cells; no flow along the edges of the domain
                e = 0 if side == 0 else n - 1
                for q in range(d + 1, self.nd):
                    for c in (-1, self.n[q] - 1):
                        w = dict(core)
                        w[q] = c + H
                        v[q][self.at(d, e, others=w)] = 0
                div = 0
                for q in [r % self.nd for r in range(d + 1, d + self.nd)]:
                    lo = dict(core)
                    lo[q] = slice(H - 1, H - 1 + self.n[q])
                    div = div + (v[q][self.at(d, e, others=lo)] - v[q][self.at(d, e, others=core)])
                x = a[self.at(d, e, others=core)] - div if side == 0 else a[self.at(d, e - 1, others=core)] + div
                for r in range(-H, -k) if side == 0 else range(n - 1 + k, n - 1 + H):
                    a[self.at(d, r, others=core)] = x

    def normal(self, v, d):
        for q in range(self.nd):
            if q == d:
                continue
            if self.bc == "cyclic":
                self.scalar(v[d], [q])
            else:
                v[d][self.at(q, -H, 0)] = 0
                v[d][self.at(q, self.n[q], self.n[q] + H)] = 0

    def sh(self, a, *by):
        """a at an offset: pairs (axis, points)."""
        for d, m in by:
            a = torch.roll(a, -m, d)
        return a

    def flux(self, p, c):
        return [x.clamp(min=0) * p + x.clamp(max=0) * self.sh(p, (d, 1)) for d, x in enumerate(c)]

    def frac(self, num, den):
        return num / (den + self.tiny)

    def antidiff(self, p, C):
        iga, tot, s, out = "iga" in self.o, "tot" in self.o, self.sh, []

        def nd4(a, b, c, e):
            return (a + b - c - e) / 4 if iga else self.frac(a + b - c - e, a + b + c + e)

        def nd2(a, b, c, e):
            return 2 * (a - b - c + e) / 4 if iga else 2 * self.frac(a - b - c + e, a + b + c + e)

        for d in range(self.nd):
            c, pr = C[d], s(p, (d, 1))
            r = c.abs() / 2 * (1 - c.abs()) * ((pr - p) if iga else 2 * self.frac(pr - p, pr + p))
            bars = []
            for q in [x % self.nd for x in range(d + 1, d + self.nd)]:
                b = (s(C[q], (d, 1)) + C[q] + s(C[q], (d, 1), (q, -1)) + s(C[q], (q, -1))) / 4
                w = [s(pr, (q, 1)), s(p, (q, 1)), s(pr, (q, -1)), s(p, (q, -1))]
                r = r - c / 2 * b * nd4(*w)
                if tot:
                    r = r + nd2(*w) * ((c.abs() - 2 * c * c) * b / 2)
                bars.append((q, b))
            if tot:
                r = r + nd2(s(p, (d, 2)), pr, p, s(p, (d, -1))) * ((3 * c * c.abs() - 2 * c ** 3 - c) / 6)
                if self.nd == 3:
                    (q1, b1), (q2, b2) = bars
                    t = [s(x, (q1, i), (q2, j)) for x in (pr, p) for i, j in ((1, 1), (-1, -1), (1, -1), (-1, 1))]
                    m = t[0] + t[1] - t[2] - t[3] + t[4] + t[5] - t[6] - t[7]
                    r = r - 2 / 3 * c * b1 * b2 * (m / 8 if iga else self.frac(m, sum(t)))
            out.append(r)
        return out

    def around(self, p, f):
        m = p
        for d in range(self.nd):
            m = f(f(m, self.sh(p, (d, 1))), self.sh(p, (d, -1)))
        return m

    def limited(self, p, c, lo, hi):
        self.along(c, True)
        for d in range(self.nd):
            self.normal(c, d)
        f = c if "iga" in self.o else self.flux(p, c)
        hi, lo = torch.maximum(hi, self.around(p, torch.maximum)), torch.minimum(lo, self.around(p, torch.minimum))
        into = sum(self.sh(x, (d, -1)).clamp(min=0) - x.clamp(max=0) for d, x in enumerate(f))
        out = sum(x.clamp(min=0) - self.sh(x, (d, -1)).clamp(max=0) for d, x in enumerate(f))
        up, dn = (hi - p) / (into + self.eps), (p - lo) / (out + self.eps)
        r = []
        for d, x in enumerate(c):
            a, b = torch.minimum(dn, self.sh(up, (d, 1))), torch.minimum(up, self.sh(dn, (d, 1)))
            r.append(x * torch.where(x > 0, a, b).clamp(max=1))
        return r

    def step(self):
        p, fct = self.p, "fct" in self.o
        self.scalar(p)
        if fct:
            lo, hi = self.around(p, torch.minimum), self.around(p, torch.maximum)
        g = unco = self.g
        for it in range(self.ni):
            if it:
                self.scalar(p)
                corr = self.antidiff(p, unco)
                if fct:
                    g = self.limited(p, corr, lo, hi)
                else:
                    g = corr
                    for d in range(self.nd):
                        self.normal(g, d)
                unco = corr
            f = g if it and "iga" in self.o else self.flux(p, g)
            p = p - sum(x - self.sh(x, (d, -1)) for d, x in enumerate(f))
        self.p = p

    def result(self):
        return self.p[tuple(slice(H, H + n) for n in self.n)].contiguous()


def exact(case, seed):
    if case["solver"] == "boussinesq":
        return None  # the pressure solve stops at a tolerance: any field within it is a result
    out = []
    for grid, (psi, adv) in _problems(case, seed):
        out.append([])
        for a in psi:
            m = _mp(case, grid, a, adv)
            for _ in range(case["nt"]):
                m.step()
            out[-1].append(m.result())
            del m
    return out if len(out) <= 32 else torch.cat([a.reshape(-1) for f in out for a in f])
