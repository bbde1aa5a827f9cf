"""Workloads of the SPH package, for timing it and for checking what it computes.

A pass is what a program does between two outputs of a run: it advances the
particles held on the device by some CheapSynchronousRK2 steps and takes the
new state (position, velocity, density, specific energy, H) into its page-
locked arrays.  `package` passes hand the state over from the host first, as
a host integrator that owns the fields does at every step, and `ensemble`
passes advance a set of independent boxes together.

Results of the mixed mode go into single-precision arrays, as snapshots of
such a run are stored: its sweeps are FP32 and its fields carry single
precision.  FP64 results are taken as they are.

exact() restates the step on explicit ghost nodes and pair lists in FP64
torch, with the kernel table rebuilt in numpy.
"""
import math

import numpy as np
import torch

from spheral_gb300 import problems
from spheral_gb300.engine import Engine

NPERH = 1.51          # smoothing lengths per spacing of every generator but the sweep box
EXTENT = 2.0          # cubic B-spline


def listed():
    return [
        # the smallest runs (unit problems, interactive use): a step is mostly launches and latency
        dict(name="box_small", kind="box", side=15, precision="fp32", steps=1, walls=True),
        # a shock tube at the resolution of the planar Sod script, with walls and grad-h
        dict(name="sod_tube", kind="sod", side=80, precision="fp32", steps=4),
        # the SPH() factory's own viscosity (limited Q) on a mid-size slab
        dict(name="kh_limited_q", kind="kh", side=41, precision="fp32", steps=2, limited=True),
        # the benchmark's Kelvin-Helmholtz slab at full size
        dict(name="kh_large", kind="kh", side=112, precision="fp32", steps=6, limited=False),
        # a homogeneous box with many neighbours and grad-h, an odd lattice
        dict(name="sweep_k100", kind="sweep", side=91, precision="fp32", steps=3, neighbors=100.0),
        # self-gravitating collapse: octree build and walk beside the hydro
        dict(name="evrard", kind="evrard", side=150001, precision="fp32", steps=2),
        # tensor smoothing scale on an anisotropic lattice
        dict(name="asph_stretched", kind="asph", side=67, precision="fp32", steps=1),
        # reproducing-kernel hydro on the smoothed slab of its own test
        dict(name="crksph_kh", kind="crksph", side=64, precision="fp32", steps=2),
        # a parameter study: uneven turbulent boxes advanced together
        dict(name="ensemble", kind="ensemble", side=38, precision="fp32", steps=2, boxes=20),
        # the package under a host integrator: state in, one step, state out
        dict(name="package_kh", kind="package", side=56, precision="fp32", steps=1),
        # all-FP64 runs, the mode used where results are compared digit by digit
        dict(name="kh_fp64", kind="kh", side=40, precision="fp64", steps=1, limited=False),
        dict(name="evrard_fp64", kind="evrard", side=30011, precision="fp64", steps=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "sod", "kh", "kh", "sweep", "evrard", "asph", "crksph", "ensemble", "package", "kh64",
                       "evrard64"])
    if kind == "box":
        return dict(kind="box", side=_log_int(rng, 14, 40), precision="fp32", steps=rng.choice([1, 2]),
                    walls=rng.random() < 0.5)
    if kind == "sod":
        return dict(kind="sod", side=2 * _log_int(rng, 32, 70), precision="fp32", steps=rng.randint(1, 5))
    if kind == "kh":
        return dict(kind="kh", side=_log_int(rng, 20, 105), precision="fp32", steps=rng.randint(1, 4),
                    limited=rng.random() < 0.5)
    if kind == "sweep":
        return dict(kind="sweep", side=_log_int(rng, 24, 110), precision="fp32", steps=rng.randint(1, 3),
                    neighbors=round(rng.uniform(32.0, 128.0), 1))
    if kind == "evrard":
        return dict(kind="evrard", side=_log_int(rng, 5000, 400000), precision="fp32", steps=rng.randint(1, 2))
    if kind == "asph":
        return dict(kind="asph", side=_log_int(rng, 20, 80), precision="fp32", steps=1)
    if kind == "crksph":
        return dict(kind="crksph", side=_log_int(rng, 20, 75), precision="fp32", steps=rng.randint(1, 2))
    if kind == "ensemble":
        return dict(kind="ensemble", side=_log_int(rng, 20, 44), precision="fp32", steps=rng.randint(1, 3),
                    boxes=rng.randint(5, 24))
    if kind == "package":
        return dict(kind="package", side=_log_int(rng, 20, 80), precision="fp32", steps=1)
    if kind == "kh64":
        return dict(kind="kh", side=_log_int(rng, 18, 52), precision="fp64", steps=1, limited=rng.random() < 0.5)
    return dict(kind="evrard", side=_log_int(rng, 4000, 60000), precision="fp64", steps=1)


# -- the problems ---------------------------------------------------------------
def _problems(case, seed):
    """The case's problems (several for an ensemble), made from the seed."""
    kind, side, seed = case["kind"], case["side"], int(seed) % (1 << 31)
    if kind == "box":
        return [problems.random_box(n_side=side, seed=seed, vel_scale=0.1, jitter=0.1,
                                    boundaries="reflecting" if case["walls"] else "periodic")]
    if kind == "sod":
        p = problems.sod(nx1=side, ny1=2 * max(12, side * 3 // 20))
        rng = np.random.default_rng(seed)
        d = np.where(p.pos[:, :1] < 1.0, 1.0, 2.0) / side     # lattice spacing of each side
        p.pos += np.clip(rng.normal(0.0, 0.02, p.pos.shape), -0.1, 0.1) * d
        return [p]
    if kind in ("kh", "package"):
        p = problems.kelvin_helmholtz(n1=side, seed=seed)
        if case.get("limited"):
            p.config.update(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0, gradh_correction=True)
        return [p]
    if kind == "sweep":
        return [problems.sweep_box(n_side=side, neighbors=case["neighbors"], seed=seed)]
    if kind == "evrard":
        return [problems.evrard(n=side, seed=seed)]
    if kind == "asph":
        return [problems.stretched_box(nx=int(round(1.25 * side)), ny=side, nz=int(round(0.8 * side)), seed=seed,
                                       jitter=0.1, vel_scale=0.1)]
    if kind == "crksph":
        p = problems.kelvin_helmholtz(n1=side, seed=seed, smooth=0.025)
        p.config.update(hydro="crksph", rk_volume="sum", xsph=False, gradh_correction=False,
                        viscosity="monaghan_gingold", Cl=1.0, Cq=1.0)
        return [p]
    if kind == "ensemble":
        lo = math.log(14.0)
        sides = [int(round(math.exp(lo + (math.log(side) - lo) * (k + 0.5) / case["boxes"])))
                 for k in range(case["boxes"])]
        return [problems.turbulent_box(s, seed * 64 + k) for k, s in enumerate(sides)]
    raise ValueError(kind)


STATE = (("pos", 3), ("vel", 3), ("rho", 1), ("eps", 1), ("H", 6))


def prepare(case, seed):
    probs = _problems(case, seed)
    total = sum(p.n for p in probs)
    pin = torch.cuda.is_available()
    host = {k: torch.zeros((total, c) if c > 1 else (total,), dtype=torch.float64, pin_memory=pin) for k, c in STATE}
    out = host
    if case["precision"] != "fp64":
        out = {k: torch.zeros_like(t, dtype=torch.float32, pin_memory=pin) for k, t in host.items()}
    engines, views, at = [], [], 0
    for p in probs:
        e = Engine.from_problem(p, precision=case["precision"])
        e.initialize()
        engines.append(e)
        views.append({k: t[at:at + p.n].numpy() for k, t in host.items()})
        at += p.n
    state = dict(case=dict(case), engines=engines, views=views, host=host, out=out)
    if case["kind"] == "package":   # the host's own fields, handed over at every step
        p = probs[0]
        state["fields"] = {k: torch.from_numpy(v).pin_memory() if pin else torch.from_numpy(v) for k, v in
                           dict(pos=p.pos, vel=p.vel, mass=p.mass, rho=p.rho, eps=p.eps, H=p.H).items()}
    return state


def run(state):
    case, engines = state["case"], state["engines"]
    if case["kind"] == "ensemble":
        Engine.ensemble_advance(engines, case["steps"])
    else:
        if case["kind"] == "package":
            engines[0].upload_state(**{k: t.numpy() for k, t in state["fields"].items()})
        for _ in range(case["steps"]):
            engines[0].step()
    for e, v in zip(engines, state["views"]):
        e.download_state(**v)
    if state["out"] is not state["host"]:
        for k, t in state["host"].items():
            state["out"][k].copy_(t)
    return state["out"]


def work(case):
    """Per step: the state read and written once (12 doubles per node each way)
    and the arithmetic of the reference's pair body, 456 operations per
    unordered pair; a walk of about 300 monopoles of 20 operations each with
    gravity.  Per pass: the state handed out (and in)."""
    kind, side = case["kind"], case["side"]
    k = case.get("neighbors", 4.0 * math.pi / 3.0 * (EXTENT * NPERH) ** 3)
    if kind in ("kh", "package", "crksph"):
        n = 1.5 * side ** 3
    elif kind == "sod":
        n = side * (2 * max(12, side * 3 // 20)) ** 2 * 1.125
    elif kind == "evrard":
        n = side
    elif kind == "asph":
        n = int(round(1.25 * side)) * side * int(round(0.8 * side))
    elif kind == "ensemble":
        lo = math.log(14.0)
        n = sum(math.exp(3.0 * (lo + (math.log(side) - lo) * (b + 0.5) / case["boxes"])) for b in range(case["boxes"]))
    else:
        n = side ** 3
    flops = case["steps"] * n * (k / 2.0 * 456.0 + (6000.0 if kind == "evrard" else 0.0))
    return {"bytes": n * 8.0 * (24.0 * case["steps"] + 14.0 + (15.0 if kind == "package" else 0.0)), "flops": flops}


# -- the same steps in plain FP64 ---------------------------------------------------
def _bspline(eta):
    w = np.where(eta < 1.0, 1.0 - 1.5 * eta ** 2 + 0.75 * eta ** 3, 0.25 * np.maximum(2.0 - eta, 0.0) ** 3)
    g = np.where(eta < 1.0, -(3.0 - 2.25 * eta) * eta, -0.75 * np.maximum(2.0 - eta, 0.0) ** 2)
    return w / math.pi, g / math.pi


class _Table:
    """Quadratic interpolants of W and dW/deta on 500 intervals, and the
    cubic Hermite lookup of nPerh from the cube root of the summed |dW/deta|."""

    def __init__(self, device, points=1000):
        m = ((points | 1) - 1) // 2
        self.step, self.m = EXTENT / m, m
        x = np.arange(2 * m + 1) * (0.5 * self.step)
        a = x[0:-2:2]
        co = []
        for y in _bspline(x):
            y0, y1, y2 = y[0:-2:2], y[1::2], y[2::2]
            c2 = 2.0 * (y0 - 2.0 * y1 + y2) / self.step ** 2
            c1 = (y2 - y0) / self.step - c2 * (2.0 * a + self.step)
            co.append(np.stack([y0 - c1 * a - c2 * a * a, c1, c2], axis=1))
        self.np_g = co[1]
        self.w, self.g = (torch.from_numpy(c).to(device) for c in co)
        self.W0 = float(co[0][0, 0])
        lo, hi = max(0.25, 1.1 / EXTENT), 64.0
        xs = np.linspace(lo, hi, points)
        self.shell = (lo, hi, np.array([self._shells(v) for v in xs]))
        ws = self._slopes(self.shell[2], (hi - lo) / (points - 1))
        wlo, whi = self.shell[2][0], self.shell[2][-1]
        targets = wlo + np.arange(points) * ((whi - wlo) / (points - 1))
        b0, b1 = np.full(points, lo), np.full(points, hi)
        for _ in range(60):
            mid = 0.5 * (b0 + b1)
            below = self._hermite(mid, lo, hi, self.shell[2], ws) < targets
            b0, b1 = np.where(below, mid, b0), np.where(below, b1, mid)
        v = 0.5 * (b0 + b1)
        v[0], v[-1] = lo, hi
        s = self._monotonic(v, self._slopes(v, (whi - wlo) / (points - 1)), (whi - wlo) / (points - 1))
        self.range, self.v, self.s = (wlo, whi), torch.from_numpy(v).to(device), torch.from_numpy(s).to(device)

    def _shells(self, nperh):
        q = np.arange(1, int(EXTENT * nperh) + 2, dtype=np.float64)
        e = np.cumsum(np.full(len(q), 1.0 / nperh))
        q, e = q[e < EXTENT], e[e < EXTENT]
        c = self.np_g[np.minimum(self.m - 1, (e / self.step).astype(np.int64))]
        return (4.0 * math.pi * np.sum(q * q * np.abs(c[:, 0] + (c[:, 1] + c[:, 2] * e) * e))) ** (1.0 / 3.0)

    @staticmethod
    def _slopes(v, h):
        n = len(v)
        A = np.zeros((n, n))
        A[np.arange(n), np.arange(n)] = 4.0
        A[np.arange(1, n - 1), np.arange(0, n - 2)] = A[np.arange(1, n - 1), np.arange(2, n)] = -0.5
        A[0, 1] = A[n - 1, n - 2] = -1.0
        r = np.empty(n)
        r[0], r[-1] = 3.0 * (v[1] - v[0]) / h, 3.0 * (v[-1] - v[-2]) / h
        r[1:-1] = 1.5 * (v[2:] - v[:-2]) / h
        return np.linalg.solve(A, r)

    @staticmethod
    def _monotonic(v, s, h):
        c, s, done = np.diff(v) / h, s.copy(), False
        for k in range(1, len(v) - 1):
            if c[k - 1] * c[k] <= 0.0:
                s[k] = 0.0
        while not done:
            done = True
            for k in range(len(v) - 1):
                a, b = s[k] / c[k], s[k + 1] / c[k]
                if a < 0.0 or b < 0.0:
                    s[k], s[k + 1], done = max(a, 0.0) * c[k], max(b, 0.0) * c[k], False
                    a, b = max(a, 0.0), max(b, 0.0)
                if a * a + b * b > 9.0:
                    t = 0.99 * 3.0 / math.sqrt(a * a + b * b)
                    s[k], s[k + 1], done = t * a * c[k], t * b * c[k], False
        return s

    @staticmethod
    def _hermite(x, lo, hi, v, s):
        lib = torch if isinstance(x, torch.Tensor) else np
        n = len(v)
        h = (hi - lo) / (n - 1)
        at = lib.clip((x - lo) / h, 0, n - 2)
        k = at.long() if lib is torch else at.astype(np.int64)
        t = lib.clip((x - lo) / h - k, 0.0, 1.0)
        t2, t3 = t * t, t * t * t
        return ((2 * t3 - 3 * t2 + 1) * v[k] + (3 * t2 - 2 * t3) * v[k + 1] +
                h * ((t3 - 2 * t2 + t) * s[k] + (t3 - t2) * s[k + 1]))

    def nperh(self, w):
        lo, hi = self.range
        y = self._hermite(w, lo, hi, self.v, self.s)
        return torch.where(w < lo, self.v[0] + self.s[0] * (w - lo), y)

    def eval(self, eta):
        k = torch.clamp((eta / self.step).long(), max=self.m - 1)
        ok = eta < EXTENT
        return [torch.where(ok, c[k, 0] + (c[k, 1] + c[k, 2] * eta) * eta, 0.0 * eta) for c in (self.w, self.g)]


def _dot(a, b):
    return (a * b).sum(-1)


def _eigenvalues(H):
    return torch.linalg.eigvalsh(H.cpu()).to(H.device)


class _Exact:
    """One problem advanced in FP64 on explicit ghost images."""

    CHUNK = 1 << 22     # pairs per piece of a sweep

    def __init__(self, p, device, table):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)
        self.T, self.dev, self.cfg, self.nl, self.bcs = table, device, p.config, p.nodelists[0], p.boundaries
        self.x, self.v, self.m, self.rho, self.u = t(p.pos), t(p.vel), t(p.mass), t(p.rho), t(p.eps)
        self.n = p.n
        self.tensor = self.cfg.get("smoothing_scale", "sph") != "sph"
        self.crk = self.cfg.get("hydro") == "crksph"
        self.h = t(p.H[:, 0])                                     # 1/h
        H = t(p.H)
        self.H = torch.stack([H[:, [0, 1, 2]], H[:, [1, 3, 4]], H[:, [2, 4, 5]]], 1) if self.tensor else None
        z = lambda *s: torch.zeros(s, dtype=torch.float64, device=device)
        n = p.n
        self.d = dict(x=z(n, 3), v=z(n, 3), rho=z(n), u=z(n), h=z(n), q=z(n), dvdx=z(n, 3, 3), grav=z(n, 3))
        self.votes = 1.0e300
        self.last = self.cfg["last_dt"]
        self.time = 0.0
        self._eos()

    def _eos(self):
        g = self.nl["gamma"]
        self.P = (g - 1.0) * self.rho * self.u
        self.c = torch.sqrt(torch.clamp(g * (g - 1.0) * self.u, min=0.0))

    # ghost images and pairs (i owned, j any image) with min(|H_i r|, |H_j r|) <= extent
    def _ghosts(self):
        hmin = _eigenvalues(self.H)[:, 0] if self.tensor else self.h
        cut = EXTENT / float(hmin.min()) * (1.0 + 1.0e-9)
        src = torch.arange(self.n, device=self.dev)
        sign = torch.ones((self.n, 3), dtype=torch.float64, device=self.dev)
        off = torch.zeros_like(sign)
        for b in self.bcs:
            a = b["axis"]
            maps = [(1.0, b["hi"] - b["lo"]), (1.0, b["lo"] - b["hi"])] if b["type"] == 0 else \
                [(-1.0, 2.0 * (b["hi"] if b.get("wall_high", 0) else b["lo"]))]
            lo, hi = b["lo"] - cut, b["hi"] + cut
            parts = [(src, sign, off)]
            for s, o in maps:
                y = s * (sign[:, a] * self.x[src, a] + off[:, a]) + o
                k = torch.nonzero((y >= lo) & (y <= hi)).flatten()
                sg, of = sign[k].clone(), off[k].clone()
                sg[:, a] *= s
                of[:, a] = s * of[:, a] + o
                parts.append((src[k], sg, of))
            src, sign, off = (torch.cat(c) for c in zip(*parts))
        return cut, src, sign, off

    def _gx(self, g):
        return self.sign[g] * self.x[self.src[g]] + self.off[g]

    def _vec(self, f, g):
        return self.sign[g] * f[self.src[g]]

    def _mat(self, f, g):
        s = self.sign[g]
        return f[self.src[g]] * s[:, :, None] * s[:, None, :]

    def _eta(self, r, i, g):
        """H_i r and H_j r."""
        if self.tensor:
            return torch.einsum("pab,pb->pa", self.H[i], r), torch.einsum("pab,pb->pa", self._mat(self.H, g), r)
        return self.h[i, None] * r, self.h[self.src[g], None] * r

    def _pairs(self):
        cut, self.src, self.sign, self.off = self._ghosts()
        y = self._gx(torch.arange(len(self.src), device=self.dev))
        lo = y.min(0).values
        edge = cut
        c = torch.floor((y - lo) / edge).long()
        nc = (c.max(0).values + 3).tolist()
        key = ((c[:, 2] + 1) * nc[1] + c[:, 1] + 1) * nc[0] + c[:, 0] + 1
        key, order = torch.sort(key)
        cells = torch.arange(nc[0] * nc[1] * nc[2] + 1, device=self.dev)
        start = torch.searchsorted(key, cells)
        self.pieces = []
        own = ((c[:self.n, 2] + 1) * nc[1] + c[:self.n, 1] + 1) * nc[0] + c[:self.n, 0] + 1
        shifts = torch.tensor([(dz * nc[1] + dy) * nc[0] + dx for dz in (-1, 0, 1) for dy in (-1, 0, 1)
                               for dx in (-1, 0, 1)], device=self.dev)
        per = max(1, int(len(key) / max(1, int((start[1:] > start[:-1]).sum()))))
        block = max(256, self.CHUNK * 4 // (27 * per))
        for s in range(0, self.n, block):
            i = torch.arange(s, min(self.n, s + block), device=self.dev)
            cc = (own[i, None] + shifts).flatten()
            cnt = start[cc + 1] - start[cc]
            base = torch.repeat_interleave(start[cc] - (torch.cumsum(cnt, 0) - cnt), cnt)
            ii = torch.repeat_interleave(i.repeat_interleave(27), cnt)
            g = order[base + torch.arange(len(base), device=self.dev)]
            r = self.x[ii] - self._gx(g)
            r2 = _dot(r, r)
            k = (r2 <= cut * cut) & (g != ii)
            ii, g, r = ii[k], g[k], r[k]
            ei, ej = self._eta(r, ii, g)
            k = torch.minimum(_dot(ei, ei), _dot(ej, ej)) <= EXTENT * EXTENT
            ii, g = ii[k], g[k]
            self.pieces += [(ii[a:a + self.CHUNK], g[a:a + self.CHUNK]) for a in range(0, len(ii), self.CHUNK)]

    def _sum(self, f, *shape):
        """Sums over the pairs of each node: f(i, g, r) gives the terms."""
        out = [torch.zeros((self.n,) + s, dtype=torch.float64, device=self.dev) for s in shape]
        for i, g in self.pieces:
            for o, v in zip(out, f(i, g, self.x[i] - self._gx(g))):
                o.index_add_(0, i, v)
        return out

    def _det(self, k=slice(None)):
        return torch.linalg.det(self.H[k]) if self.tensor else self.h[k] ** 3

    def _density(self):
        def terms(i, g, r):
            ej = self._eta(r, i, g)[1]
            j = self.src[g]
            w = self.T.eval(ej.norm(dim=1))[0] * det[j]
            if self.crk:
                vw = self.V[j] * w
                return vw, self.m[j] * vw, self.V[j] * vw
            return (self.m[j] * w,)
        det = self._det()
        if not self.crk:
            self.rho = self.m * det * self.T.W0 + self._sum(terms, ())[0]
            return
        self.V = 1.0 / (det * (self._sum(lambda i, g, r: (self.T.eval(self.h[i] * r.norm(dim=1))[0],), ())[0] + self.T.W0))
        self.V = torch.minimum(self.V, 4.0 / 3.0 * math.pi * (0.5 * EXTENT) ** 3 / det)
        w, mw, vw = self._sum(terms, (), (), ())
        s = self.V * det * self.T.W0
        w = w + s
        rho = (mw + self.m * s) / (w * ((vw + self.V * s) / w))
        self.rho = torch.maximum(torch.clamp(rho, max=self.nl["rhoMax"]), torch.clamp(0.1 * self.m * det, min=self.nl["rhoMin"]))

    def _dt(self, left):
        tiny, nperh = 2.220446049250313e-16, self.nl["nPerh"]
        hx = _eigenvalues(self.H)[:, 2] if self.tensor else self.h
        ns, vm = 1.0 / (hx * nperh), self.v.norm(dim=1)
        div = torch.einsum("naa->n", self.d["dvdx"])
        lim = [ns / (self.c + tiny), ns / (torch.sqrt(self.d["q"] / self.rho) + tiny), 1.0 / (div.abs() + tiny),
               0.1 * torch.maximum(ns / (vm + tiny), vm / (self.d["v"].norm(dim=1) + tiny))]
        dt = min(float(x.min()) for x in lim)
        for i, g in self.pieces:
            s = torch.minimum(ns[i], ns[self.src[g]])
            dt = min(dt, float((s / torch.clamp((self.v[i] - self._vec(self.v, g)).norm(dim=1), min=1e-30)).min()))
        dt *= self.cfg["cfl"]
        if self.cfg.get("gravity"):
            dt = min(dt, self.cfg["ftimestep"] * self.votes)
        dt = min(dt, self.cfg["dt_max"], left, self.cfg["dt_growth"] * self.last)
        return max(dt, self.cfg["dt_min"])

    def _gravity(self):
        x, s2, a = self.x, self.cfg["softening"] ** 2, torch.zeros_like(self.x)
        piece = max(1, (1 << 27) // self.n)
        for s in range(0, self.n, piece):
            r = [x[None, :, k] - x[s:s + piece, None, k] for k in range(3)]
            q = r[0] * r[0] + r[1] * r[1] + r[2] * r[2]
            f = torch.where(q > 1e-10 * s2, self.m / (q + s2) * torch.rsqrt(torch.clamp(q, min=1e-300)), 0.0 * q)
            for k in range(3):
                a[s:s + piece, k] = (f * r[k]).sum(1)
        self.votes = float(torch.sqrt(self.cfg["softening"] / a.norm(dim=1)).min()) / math.sqrt(self.cfg["G"])
        return self.cfg["G"] * a

    def _corrections(self):
        """C and dC/dx of the LinearOrder reproducing kernels."""
        def terms(i, g, r):
            j = self.src[g]
            W, G = self.T.eval(self.h[j] * r.norm(dim=1))
            w = W * self.h[j] ** 3
            dw = (G * self.h[j] ** 4 / r.norm(dim=1).clamp(min=1e-300))[:, None] * r
            P = torch.cat([torch.ones_like(r[:, :1]), r], 1)
            PP = P[:, :, None] * P[:, None, :]
            v = self.V[j]
            dM = PP[:, None] * (v[:, None] * dw)[:, :, None, None]
            for a in range(3):
                dM[:, a, 1 + a, :] += (v * w)[:, None] * P
                dM[:, a, :, 1 + a] += (v * w)[:, None] * P
            return PP * (v * w)[:, None, None], dM
        M, dM = self._sum(terms, (4, 4), (3, 4, 4))
        W, G = (float(c[0, 0]) for c in (self.T.w, self.T.g))
        M[:, 0, 0] += self.V * self.h ** 3 * W
        dM[:, 0, 0, 0] += self.V * self.h ** 4 * G
        for a in range(3):
            dM[:, a, 0, 1 + a] += self.V * self.h ** 3 * W
            dM[:, a, 1 + a, 0] += self.V * self.h ** 3 * W
        e = torch.zeros((self.n, 4), dtype=torch.float64, device=self.dev)
        e[:, 0] = 1.0
        C = torch.linalg.solve(M, e)
        D = torch.linalg.solve(M, -torch.einsum("ndkl,nl->nkd", dM, C))
        return C, D.transpose(1, 2).contiguous()

    def _reproduce(self, C, D, x, h):
        """W^R(x) with its gradient (base kernel of 1/h, coefficients C, D)."""
        r = x.norm(dim=1)
        W, G = self.T.eval(h * r)
        w = W * h ** 3
        dw = (G * h ** 4 / r.clamp(min=1e-300))[:, None] * x
        cp = C[:, 0] + _dot(C[:, 1:], x)
        dp = C[:, 1:] + D[:, :, 0] + torch.einsum("pdk,pk->pd", D[:, :, 1:], x)
        return cp * w, cp[:, None] * dw + dp * w[:, None], G

    def _force(self, i, g, r):
        """Pair acceleration of i, and what the derivative sums need."""
        c, j = self.cfg, self.src[g]
        ei, ej = self._eta(r, i, g)
        ni, nj = ei.norm(dim=1), ej.norm(dim=1)
        vij = self.v[i] - self._vec(self.v, g)
        vq = vij
        if c.get("viscosity") == "limited_monaghan_gingold":
            hx = 0.5 * r
            ai, aj = torch.einsum("pab,pb->pa", self.Q[i], hx), torch.einsum("pab,pb->pa", self._mat(self.Q, g), hx)
            gi, gj = _dot(ai, hx), _dot(aj, hx)
            safe = lambda y: torch.where(y < 0, -1.0, 1.0) * y.abs().clamp(min=1e-30)
            q = torch.minimum(gi / safe(gj), gj / safe(gi))
            phi = torch.where(q > 0, 4.0 * q / (1.0 + q) ** 2, 0.0 * q)
            crit, fold = 1.0 / self.nl["nPerh"], 0.2 / self.nl["nPerh"]
            eta = torch.minimum(ni, nj)
            phi = torch.where(eta < crit, phi * torch.exp(-((eta - crit) / fold) ** 2), phi)
            vq = vij - phi[:, None] * (ai + aj)
        mui = torch.clamp(_dot(vq, ei) / (ni * ni + 1e-2), max=0.0)
        muj = torch.clamp(_dot(vq, ej) / (nj * nj + 1e-2), max=0.0)
        qi = -c["Cl"] * self.c[i] * mui + c["Cq"] * mui * mui
        qj = -c["Cl"] * self.c[j] * muj + c["Cq"] * muj * muj
        if self.crk:
            Wj, gj, _ = self._reproduce(self.C[i], self.D[i], r, self.h[j])
            s = self.sign[g]
            Cj = self.C[j] * torch.cat([torch.ones_like(s[:, :1]), s], 1)
            Dj = self.D[j] * s[:, :, None] * torch.cat([torch.ones_like(s[:, :1]), s], 1)[:, None, :]
            _, gi, Gi = self._reproduce(Cj, Dj, -r, self.h[i])
            f = 0.5 * self.V[i] * self.V[j]
            dg = gj - gi
            a = -(f * (self.P[i] + self.P[j] + self.rho[i] * qi + self.rho[j] * qj) / self.m[i])[:, None] * dg
            de = f * (self.P[j] + self.rho[j] * qj) * _dot(vij, dg) / self.m[i]
            return a, de, -(self.V[j, None] * vij)[:, :, None] * gj[:, None, :], 4.0 * self.rho[i] * qi, Gi
        det = self.det
        Wi, Gi = self.T.eval(ni)
        Gj = self.T.eval(nj)[1]
        ui, uj = ei / ni.clamp(min=1e-30)[:, None], ej / nj.clamp(min=1e-30)[:, None]
        if self.tensor:
            gi = (det[i] * Gi)[:, None] * torch.einsum("pab,pb->pa", self.H[i], ui)
            gj = (det[j] * Gj)[:, None] * torch.einsum("pab,pb->pa", self._mat(self.H, g), uj)
        else:
            gi, gj = (det[i] * Gi * self.h[i])[:, None] * ui, (det[j] * Gj * self.h[j])[:, None] * uj
        Pi = self.P[i] / (self.om[i] * self.rho[i] ** 2) + 0.5 * qi / self.rho[i]
        Pj = self.P[j] / (self.om[j] * self.rho[j] ** 2) + 0.5 * qj / self.rho[j]
        a = -self.m[j, None] * (Pi[:, None] * gi + Pj[:, None] * gj)
        return a, self.m[j] * Pi * _dot(vij, gi), -self.m[j, None, None] * vij[:, :, None] * gi[:, None, :], \
            self.rho[i] * qi, Gi, -self.m[j, None, None] * r[:, :, None] * gi[:, None, :]

    def _derivatives(self):
        n = self.n
        self.det = self._det()
        if self.crk:
            self.C, self.D = self._corrections()
        self.om = torch.ones(n, dtype=torch.float64, device=self.dev)
        if self.cfg["gradh_correction"]:
            def omega(i, g, r):
                e = self._eta(r, i, g)[0].norm(dim=1)
                W, G = self.T.eval(e)
                return W, e * G
            w, eg = self._sum(omega, (), ())
            self.om = torch.clamp(-eg / (3.0 * (w + self.T.W0)), min=1e-30)
        q = torch.zeros(n, dtype=torch.float64, device=self.dev)
        cnt = torch.zeros(n, dtype=torch.float64, device=self.dev)

        def terms(i, g, r):
            f = self._force(i, g, r)
            q.scatter_reduce_(0, i, f[3], "amax")
            cnt.index_add_(0, i, torch.ones_like(f[1]))
            return f[:3] + (f[4].abs(),) + f[5:]
        sums = self._sum(terms, (3,), (), (3, 3), (), *(() if self.crk else ((3, 3),)))
        d = self.d
        d["v"], d["u"], D, m0 = sums[:4]
        if not self.crk:
            M = sums[4]
            ok = (torch.linalg.det(M).abs() > 1e-10) & (cnt > 8)
            eye = torch.eye(3, dtype=torch.float64, device=self.dev)
            D = torch.where(ok[:, None, None], D @ torch.linalg.inv(torch.where(ok[:, None, None], M, eye)),
                            D / self.rho[:, None, None])
        tr = torch.einsum("naa->n", D)
        d["dvdx"], d["q"], d["x"], d["rho"] = D, q, self.v.clone(), -self.rho * tr
        if self.cfg.get("gravity"):
            d["grav"] = self._gravity()
        if not self.tensor:
            d["h"] = -self.h / 3.0 * tr
            nperh = self.nl["nPerh"]
            s = (nperh / (torch.clamp(self.T.nperh(m0 ** (1.0 / 3.0)), min=0.0) + 1e-30)).clamp(0.25, 4.0)
            a = torch.where(s < 1.0, 0.4 * (1.0 + s * s), 0.4 * (1.0 + 1.0 / s ** 3))
            self.ideal = 1.0 / ((1.0 - a + a * s) / self.h).clamp(self.nl["hmin"], self.nl["hmax"])

    def _update(self, dt, mid):
        d = self.d
        if mid:
            self.u = self.u + dt * d["u"]
        self.x = self.x + dt * d["x"]
        self.v = self.v + dt * (d["v"] + d["grav"])
        if self.crk:
            rho = self.rho + dt * d["rho"]
            V = self.V - dt * self.m / (rho * rho) * d["rho"]
            self.V = torch.maximum(0.5 * self.m / rho, torch.minimum(4.0 * math.pi / (3.0 * self.h ** 3), V))
        self.rho = (self.rho + dt * d["rho"]).clamp(self.nl["rhoMin"], self.nl["rhoMax"])
        if not self.tensor:
            self.h = (self.h + dt * d["h"] if mid else self.ideal).clamp(1.0 / self.nl["hmax"], 1.0 / self.nl["hmin"])
        self._eos()

    def step(self):
        self._pairs()
        self._density()
        dt = self._dt(1.0e300)
        keep = (self.x, self.v, self.rho, self.u, self.h)
        self.Q = self.d["dvdx"]
        self._update(0.5 * dt, True)
        self._derivatives()
        if self.crk:
            V = self.V
        d0, w = self.d["u"], torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        v12 = keep[1] + 0.5 * dt * self.d["v"]
        for i, g in self.pieces:
            a = self._force(i, g, self.x[i] - self._gx(g))[0]
            du = _dot(self._vec(v12, g) - v12[i], a)
            sg = torch.where(du < 0.0, -1.0, 1.0)
            wi, wj = ((d0[k] * sg).clamp(min=2.220446049250313e-16) for k in (i, self.src[g]))
            w.index_add_(0, i, wi / (wi + wj) * du)
        self.x, self.v, self.rho, self.u, self.h = keep
        if self.crk:
            self.V = V
        self.u = self.u + dt * w
        self._update(dt, False)
        for b in self.bcs:
            x, a = self.x[:, b["axis"]], b["axis"]
            if b["type"] == 0:
                self.x[:, a] = torch.where(x < b["lo"], x + (b["hi"] - b["lo"]), torch.where(x > b["hi"], x - (b["hi"] - b["lo"]), x))
            else:
                out = x > b["hi"] if b.get("wall_high", 0) else x < b["lo"]
                self.x[:, a] = torch.where(out, 2.0 * (b["hi"] if b.get("wall_high", 0) else b["lo"]) - x, x)
                self.v[:, a] = torch.where(out, -self.v[:, a], self.v[:, a])
        self.last = dt


def exact(case, seed):
    """run()'s state for these inputs; H of the tensor smoothing scale is left out."""
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    table = _Table(device)
    parts = []
    for p in _problems(case, seed):
        e = _Exact(p, device, table)
        for _ in range(case["steps"]):
            e.step()
        H = None
        if not e.tensor:
            H = torch.zeros((e.n, 6), dtype=torch.float64, device=device)
            H[:, [0, 3, 5]] = e.h[:, None]
        parts.append(dict(pos=e.x, vel=e.v, rho=e.rho, eps=e.u, H=H))
    return {k: None if parts[0][k] is None else torch.cat([q[k] for q in parts]) for k, _ in STATE}
