"""Timed cases of the DAW redatuming library: what is run, on which inputs,
and what it computes in 64 bits.

A case is one call of a public entry point of the host mirror (host arrays in
and out, as the reference's routines take them) on a model, an acquisition
and data made from a seed.  The grids, spreads and record lengths are those
of the benchmark configurations (151x461 h=20, 751x2301 h=4, 2001x8001 h=5;
package file synthetic.py), with shorter records where a whole one would take
minutes, and ragged sizes between them.  `draw` gives further cases of the
same ranges.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "model-based-seismic-data-redatuming-with-daws_b200")


def _package():
    """The package directory (its name is not a Python identifier) as daw_b200."""
    if "daw_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "daw_b200", os.path.join(_PKG, "__init__.py"), submodule_search_locations=[_PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["daw_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["daw_b200"]


def _case(name, kind, n1, n2, npml, h, dt, f0, nt, nr, nshot=1, maxiter=0, history=16,
          density=False, checkpoint=0, wavefield=False):
    c = dict(kind=kind, n1=n1, n2=n2, npml=npml, h=h, dt=dt, f0=f0, nt=nt, nr=nr, nshot=nshot,
             maxiter=maxiter, history=history, density=density, checkpoint=checkpoint,
             wavefield=wavefield)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The band pass of a redatumed gather by itself: 230 datum traces of 2000 samples.
        _case("filter_2000x230", "filter", 151, 461, 20, 20.0, 0.0015, 10.0, 2000, 230),
        # The smallest simulation a user starts: one short shot on the small model.
        _case("forward_151x461", "forward", 151, 461, 20, 20.0, 0.0015, 10.0, 400, 230),
        # Mode 0 over several shots of uneven length (observed data of a survey).
        _case("forward_shots_751x2301", "forward", 751, 2301, 40, 4.0, 0.0004, 15.0, 450, 576,
              nshot=4),
        # One G G^T application, the operator everything iterates, with FP32 histories.
        _case("ggt_151x461_fp32", "ggt", 151, 461, 20, 20.0, 0.0015, 10.0, 1000, 230, history=32),
        # The same on the main benchmark grid with the default FP16 histories.
        _case("ggt_751x2301", "ggt", 751, 2301, 40, 4.0, 0.0004, 15.0, 1200, 576),
        # The largest grid (one shot fills the device).
        _case("ggt_2001x8001", "ggt", 2001, 8001, 50, 5.0, 0.0004, 20.0, 50, 1200),
        # Histories kept in windows, as a record too long for the device has them.
        _case("ggt_window_647x1533", "ggt", 647, 1533, 33, 5.0, 0.0005, 12.0, 450, 301,
              checkpoint=150),
        # The final simulation with the wavefield a user writes to disk (oio = 1).
        _case("esource_wavefield_151x461", "esource", 151, 461, 20, 20.0, 0.0015, 10.0, 250, 230,
              wavefield=True),
        # MINRES by itself on a ragged mid-sized model.
        _case("minres_301x703", "minres", 301, 703, 25, 10.0, 0.0008, 10.0, 750, 157, maxiter=8),
        # The whole pipeline of one shot on the small model (10 iterations, as configured there).
        _case("shot_151x461", "shots", 151, 461, 20, 20.0, 0.0015, 10.0, 600, 230, maxiter=10),
        # The headline work: uneven shots of the 751x2301 model through the whole pipeline.
        _case("shots_751x2301", "shots", 751, 2301, 40, 4.0, 0.0004, 15.0, 640, 576, nshot=3,
              maxiter=3),
        # A shot with Gardner's density.
        _case("shot_density_751x2301", "shots", 751, 2301, 40, 4.0, 0.0004, 15.0, 300, 400,
              maxiter=2, density=True),
    ]


# Simulations of one pass, in time loops of the record.
def _sims(case):
    it = case["maxiter"]
    return {"filter": 0, "forward": 1, "ggt": 2, "esource": 2, "minres": 2 * (it + 2),
            "shots": 3 + 2 * (it + 2)}[case["kind"]]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["filter", "forward", "forward", "ggt", "ggt", "ggt", "esource", "minres",
                       "minres", "shots", "shots", "shots"])
    if kind == "filter":
        return _case(None, kind, 151, 461, 20, 20.0, rng.choice([0.0004, 0.001, 0.0015, 0.002]),
                     10.0, _log_int(rng, 700, 10000), _log_int(rng, 24, 600))
    h = rng.choice([4.0, 5.0, 10.0, 20.0])
    n1 = _log_int(rng, 101, 760)
    n2 = max(n1, _log_int(rng, 201, 2310))
    npml = rng.randint(20, 45)
    dt = round(0.45 * h / 5500.0, 5)
    f0 = round(1500.0 / (h * rng.uniform(12.0, 25.0)), 1)
    nr = _log_int(rng, 40, max(60, n2 // 4))
    nshot = {"forward": rng.choice([1, 2, 4, 6]), "shots": rng.choice([1, 1, 2, 3])}.get(kind, 1)
    maxiter = {"minres": rng.randint(2, 8), "shots": rng.randint(1, 4)}.get(kind, 0)
    c = _case(None, kind, n1, n2, npml, h, dt, f0, 0, nr, nshot, maxiter,
              history=rng.choice([16, 16, 16, 32]) if kind != "forward" else 16,
              density=rng.random() < 0.2)
    # the record: 120 .. 1500 steps, as long as a budget of point updates allows
    points = (n1 + 2 * npml) * (n2 + 2 * npml) * nshot * max(1, _sims(c))
    # and long enough for the wavelet to leave the source
    lo = max(120, int(1.8 / (f0 * dt)))
    c["nt"] = _log_int(rng, lo, max(lo + 30, min(1500, 2.5e10 / points)))
    if kind == "ggt" and rng.random() < 0.25:
        c["checkpoint"] = max(20, c["nt"] // rng.randint(2, 5))
    if kind == "esource" and n1 * n2 * c["nt"] < 25_000_000:
        c["wavefield"] = True
    return c


# ---------------------------------------------------------------------------
# Inputs (from the seed alone)
# ---------------------------------------------------------------------------
def _ricker(t, f0):
    a = (np.pi * f0 * t) ** 2
    return (1.0 - 2.0 * a) * np.exp(-a)


def _model(case, rng):
    """A velocity trend with dipping, faulted layers: 1500 .. 5500 m/s (4000 for h = 20)."""
    n1, n2 = case["n1"], case["n2"]
    vmax = 4000.0 if case["h"] >= 20.0 else 5500.0
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    z = torch.linspace(0.0, 1.0, n1, device=dev)[:, None]
    x = torch.linspace(0.0, 1.0, n2, device=dev)[None, :]
    v = 1500.0 + (vmax - 1500.0) * z ** 0.8 + 0.0 * x
    for _ in range(6):
        depth = rng.uniform(0.1, 0.9) + rng.uniform(-0.1, 0.1) * (x - 0.5)
        depth = depth + rng.uniform(0.0, 0.05) * (x > rng.uniform(0.2, 0.8))
        v = v + rng.uniform(-150.0, 200.0) * (z > depth)
    return np.asfortranarray(v.clamp(1480.0, vmax).float().cpu().numpy())


def _events(case, rng, nt, xs, xr):
    """Band-limited reflection data: hyperbolic events, (nt, nr)."""
    t = (np.arange(nt) * case["dt"])[:, None]
    d = np.zeros((nt, len(xr)))
    span = nt * case["dt"]
    for _ in range(4):
        t0, v = rng.uniform(0.15, 0.8) * span, rng.uniform(1500.0, 3500.0)
        tau = np.sqrt(t0 ** 2 + ((xr - xs) / v) ** 2)[None, :]
        d += rng.uniform(-1.0, 1.0) * _ricker(t - tau, case["f0"])
    return np.asfortranarray(d.astype(np.float32))


def _inputs(case, seed):
    """Host arrays of the case: model, positions, wavelets and data of every shot."""
    rng = np.random.default_rng(seed)
    h, n1, n2, nr = case["h"], case["n1"], case["n2"], case["nr"]
    inp = dict(vp=_model(case, rng) if case["kind"] != "filter" else None, shots=[])
    if case["density"]:
        inp["rho"] = np.asfortranarray((0.31 * inp["vp"].astype(np.float64) ** 0.25)
                                       .astype(np.float32))
    xmax = (n2 - 1) * h
    # the datum, at a depth that the waves reach within the record
    depth = min(0.4 * (n1 - 1), 525.0 * (case["nt"] - (case["nshot"] - 1) * case["nt"] // 6)
                * case["dt"] / h)
    inp["datum"] = np.stack([np.full(nr, max(5, round(depth)) * h), np.linspace(0, xmax, nr)],
                            1).astype(np.float32)
    for k in range(case["nshot"]):
        nt = case["nt"] - (k * case["nt"]) // 6   # uneven record lengths and spreads
        n = max(4, nr - (k * nr) // 5)
        xs = float(np.float32(rng.uniform(0.2, 0.8) * xmax))
        length = n / nr * xmax  # a spread around the source
        lo = min(max(xs - rng.uniform(0.2, 0.8) * length, 0.0), xmax - length)
        xr = lo + np.linspace(0.0, length, n)
        t = np.arange(nt) * case["dt"] - 1.2 / case["f0"]
        inp["shots"].append(dict(
            nt=nt, src=np.array([[2.0 * h, xs]], np.float32),
            rec=np.stack([np.full(n, 3.0 * h), xr], 1).astype(np.float32),
            s=(_ricker(t, case["f0"]) * rng.uniform(0.5, 2.0) / (h * h)).astype(np.float32),
            data=_events(case, rng, nt, xs, xr)))
    return inp


def _band(case):
    f0 = case["f0"]
    return (0.5 * f0, 2.5 * f0, 0.5 * f0, 0.5 * f0)


MU, RTOL = 1e-2, 0.0


def prepare(case, seed):
    """A handle with its model, and the host arrays of the call."""
    D = _package()
    inp = _inputs(case, seed)
    if case["kind"] == "filter":
        return dict(case=case, handle=D.Handle(0), data=inp["shots"][0]["data"])
    h = D.Handle(0, preset="mixed", history=1 if case["history"] == 16 else 0,
                 checkpoint=case["checkpoint"])
    h.set_model(inp["vp"], case["npml"], case["h"], case["dt"], 1, rho=inp.get("rho"))
    tab = lambda pos: D.subacqui(pos, case["h"], case["npml"], 1)  # noqa: E731
    if case["kind"] == "shots":
        h.set_datum(tab(inp["datum"]))
    shots = []
    for sh in inp["shots"]:
        shots.append(dict(nt=sh["nt"], s=sh["s"], src=tab(sh["src"])[0], rec=tab(sh["rec"]),
                          dobs=sh["data"], mu=MU, maxiter=case["maxiter"], rtol=RTOL,
                          band=_band(case)))
    return dict(case=case, handle=h, shots=shots)


def run(state):
    case, h = state["case"], state["handle"]
    kind = case["kind"]
    if kind == "filter":
        return h.filmartin2d(state["data"], case["dt"], *_band(case))[0]
    shots = state["shots"]
    sh = shots[0]
    if kind == "forward":
        if len(shots) == 1:
            return h.submodeling(sh["s"], sh["src"], sh["rec"])[0]
        return h.submodeling_shots(shots)
    if kind == "ggt":
        return h.submodeling_adjoint_esource_data(sh["dobs"], sh["rec"])
    if kind == "esource":
        sis, wf, cost = h.submodeling_adjoint_esource(sh["dobs"], sh["rec"],
                                                      wavefield=case["wavefield"])
        return dict(sis=sis, cost=cost, **({"wavefield": wf} if case["wavefield"] else {}))
    if kind == "minres":
        x, info = h.sublinearminres(sh["dobs"], sh["rec"], MU, case["maxiter"], RTOL)
        return dict(x=x, shift=info["shift"], rnorm=info["rnorm"], anorm=info["anorm"])
    out = []
    for r in h.shots(shots):
        out.append({k: r[k] for k in ("datar", "deltadr", "deltade", "dataesc", "datae",
                                      "redatumed_raw", "redatumed")})
    return out


def work(case):
    """Inputs read once, outputs written once; stencil operations of the time
    loops (30 per point and step) or of the filter's transforms."""
    nt, nr = case["nt"], case["nr"]
    if case["kind"] == "filter":
        nto = 1 << max(3, (nt - 1).bit_length())
        return dict(bytes=8.0 * nt * nr, flops=2 * 2.5 * nto * math.log2(nto) * nr)
    points = float((case["n1"] + 2 * case["npml"]) * (case["n2"] + 2 * case["npml"]))
    steps, data = 0, 0
    for k in range(case["nshot"]):
        n = nt - (k * nt) // 6
        r = max(4, nr - (k * nr) // 5)
        steps += n * _sims(case)
        io = {"forward": 1, "ggt": 2, "esource": 2, "minres": 2, "shots": 6}[case["kind"]]
        data += 4.0 * n * (r * io + (2 * nr if case["kind"] == "shots" else 0))
    grids = 4.0 * case["n1"] * case["n2"] * (2 if case["density"] else 1)
    if case["wavefield"]:
        data += 4.0 * case["n1"] * case["n2"] * nt
    return dict(bytes=grids + data, flops=30.0 * points * steps)


# ---------------------------------------------------------------------------
# The same in 64 bits, with torch
# ---------------------------------------------------------------------------
_RAD = 10
_F64 = torch.float64


def _bessel_i0(x):
    """Abramowitz & Stegun 9.8.1 / 9.8.2, the polynomials that define the tables."""
    ax = abs(x)
    if ax < 3.75:
        y = (x / 3.75) ** 2
        return 1.0 + y * (3.5156229 + y * (3.0899424 + y * (1.2067492 + y * (
            0.2659732 + y * (0.0360768 + y * 0.0045813)))))
    y = 3.75 / ax
    return math.exp(ax) / math.sqrt(ax) * (0.39894228 + y * (0.01328592 + y * (0.00225319 + y * (
        -0.00157565 + y * (0.00916281 + y * (-0.02057706 + y * (0.02635537 + y * (
            -0.01647633 + y * 0.00392377))))))))


def _kws(ia):
    """Kaiser-windowed sinc of sub-grid position ia (1 .. 100), taps -10 .. 10."""
    c = np.zeros(2 * _RAD + 1)
    for n in range(-_RAD, _RAD + 1):
        x = n + 0.5 - (ia - 1) / 100.0
        if abs(x) < 1e-12:
            c[n + _RAD] = 1.0
        elif abs(x) <= _RAD:
            kaiser = _bessel_i0(14.18 * math.sqrt(1.0 - x * x / _RAD ** 2)) / _bessel_i0(14.18)
            c[n + _RAD] = kaiser * math.sin(math.pi * x) / (math.pi * x)
    return c


class _Stations:
    """Interpolation of (z, x) positions on an array of n1 x n2 points whose
    first point is `pad` points outside the physical grid; the taps above the
    free surface are folded back with the opposite sign."""

    def __init__(self, pos, h, n1, n2, pad, dev):
        f = np.float32
        nint = lambda v: int(math.floor(abs(float(v)) + 0.5)) * (1 if v >= 0 else -1)  # noqa: E731
        idx = np.zeros((len(pos), 441), np.int64)
        coef = np.zeros((len(pos), 441))
        tabs = {}
        for r, p in enumerate(np.asarray(pos, f)):
            i, c = [], []
            for d in range(2):
                q = nint(p[d] / f(h))
                alpha = (f(q) * f(h) - p[d]) / f(h)
                ia = min(nint((f(0.5) - alpha) * f(100)) + 1, 100)
                if ia not in tabs:
                    tabs[ia] = _kws(ia)
                i.append(q + pad)
                c.append(tabs[ia])
            tile = np.outer(c[0], c[1])
            nfs = max(_RAD - nint(p[0] / f(h)), 0)
            if nfs > 0:
                m = _RAD - (_RAD - nfs)  # tile row on the free surface
                folded = tile.copy()
                folded[m] = 0.0
                for k in range(1, nfs + 1):
                    folded[m + k] = tile[m + k] - tile[m - k]
                tile = folded
            a = i[0] + np.arange(-_RAD, _RAD + 1)[:, None] + 0 * np.arange(21)[None, :]
            b = i[1] + np.arange(-_RAD, _RAD + 1)[None, :] + 0 * np.arange(21)[:, None]
            ok = (a >= 0) & (a < n1) & (b >= 0) & (b < n2)
            idx[r] = np.where(ok, a * n2 + b, 0).ravel()
            coef[r] = np.where(ok, tile, 0.0).ravel()
        self.idx = torch.from_numpy(idx).to(dev)
        self.coef = torch.from_numpy(coef).to(dev)

    def gather(self, f):
        return (f.reshape(-1)[self.idx] * self.coef).sum(1)

    def add(self, f, amp):
        f.view(-1).index_add_(0, self.idx.view(-1), (self.coef * amp[:, None]).view(-1))


class _Wave:
    """Staggered-grid simulations of one model in 64 bits."""

    A0, A1 = 1.125, -1.0 / 24.0

    def __init__(self, case, inp):
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        n1, n2, m = case["n1"], case["n2"], case["npml"]
        self.n1, self.n2, self.m = n1, n2, m
        self.h, self.dt = float(np.float32(case["h"])), float(np.float32(case["dt"]))

        def extend(a):
            i = torch.arange(n1 + 2 * m).sub(m).clamp(0, n1 - 1)
            j = torch.arange(n2 + 2 * m).sub(m).clamp(0, n2 - 1)
            return torch.from_numpy(a.astype(np.float64)).to(dev)[i.to(dev)][:, j.to(dev)]

        rho = extend(inp["rho"]) if "rho" in inp else None
        self.kap = extend(inp["vp"]) ** 2 * (rho if rho is not None else 1.0)
        self.bu = 1.0 / rho if rho is not None else None

        def sponge(n, shift):
            d = torch.ones(n + 2 * m, dtype=_F64, device=dev)
            k = torch.arange(m, dtype=_F64, device=dev)  # distance from the physical grid
            if shift:
                d[:m - 1] = torch.exp(-(0.12 * (k[:m - 1] + 0.5)) ** 2).flip(0)
                d[m + n:] = torch.exp(-(0.12 * (k + 0.5)) ** 2)
            else:
                d[:m] = torch.exp(-(0.12 * k) ** 2).flip(0)
                d[m + n:] = torch.exp(-(0.12 * k) ** 2)
            return d

        self.a1, self.a2 = sponge(n1, False)[:, None], sponge(n2, False)[None, :]
        self.b1, self.b2 = sponge(n1, True)[:, None], sponge(n2, True)[None, :]
        q = self.dt / self.h
        bu1 = bu2 = torch.ones(1, 1, dtype=_F64, device=dev)
        if rho is not None:
            bu1, bu2 = self.bu.clone(), self.bu.clone()
            bu1[:-1] = 0.5 * (self.bu[1:] + self.bu[:-1])
            bu2[:, :-1] = 0.5 * (self.bu[:, 1:] + self.bu[:, :-1])
        self.kw1, self.kw2 = q * self.kap * self.a1.sqrt(), q * self.kap * self.a2.sqrt()
        self.bw1, self.bw2 = q * bu1 * self.b1.sqrt(), q * bu2 * self.b2.sqrt()

    def zeros(self):
        return [torch.zeros_like(self.kap) for _ in range(4)]  # px, pz, vx, vz

    def interior(self, f, cut=0):
        m = self.m
        return f[m + cut:m + self.n1 - cut, m + cut:m + self.n2 - cut]

    def p_step(self, st, off, sign):
        px, pz, vx, vz = st
        N1, N2 = px.shape
        I, J = slice(2, N1 - off), slice(2, N2 - off)
        s = lambda f, d, k: f.narrow(d, 2 + k, f.shape[d] - off - 2)  # noqa: E731
        X, Z = vx[I], vz[:, J]
        dx = self.A0 * (s(X, 1, 0) - s(X, 1, -1)) + self.A1 * (s(X, 1, 1) - s(X, 1, -2))
        dz = self.A0 * (s(Z, 0, 0) - s(Z, 0, -1)) + self.A1 * (s(Z, 0, 1) - s(Z, 0, -2))
        px[I, J] = self.a2[:, J] * px[I, J] + sign * self.kw2[I, J] * dx
        pz[I, J] = self.a1[I] * pz[I, J] + sign * self.kw1[I, J] * dz

    def p_sum(self, st):
        p = st[0] + st[1]
        p[:self.m + 1] = 0.0
        return p

    def v_step(self, st, p, off, sign):
        _, _, vx, vz = st
        N1, N2 = vx.shape
        I, J = slice(2, N1 - off), slice(2, N2 - off)
        s = lambda f, d, k: f.narrow(d, 2 + k, f.shape[d] - off - 2)  # noqa: E731
        X, Z = p[I], p[:, J]
        dx = self.A0 * (s(X, 1, 1) - s(X, 1, 0)) + self.A1 * (s(X, 1, 2) - s(X, 1, -1))
        dz = self.A0 * (s(Z, 0, 1) - s(Z, 0, 0)) + self.A1 * (s(Z, 0, 2) - s(Z, 0, -1))
        vx[I, J] = self.b2[:, J] * vx[I, J] + sign * self.bw2.expand_as(vx)[I, J] * dx
        vz[I, J] = self.b1[I] * vz[I, J] + sign * self.bw1.expand_as(vz)[I, J] * dz

    def surface(self, st):
        st[3][self.m - 1] = st[3][self.m]

    def stations(self, pos):
        return _Stations(pos, self.h, self.n1 + 2 * self.m, self.n2 + 2 * self.m, self.m, self.dev)

    def forward(self, s, src, rec, datum=None):
        st, out, red = self.zeros(), [], []
        kap_dt = self.kap.reshape(-1)[src.idx] * self.dt * src.coef
        for a in s.astype(np.float64):
            self.p_step(st, 2, 1.0)
            st[0].view(-1).index_add_(0, src.idx.view(-1), (kap_dt * a).view(-1))
            p = self.p_sum(st)
            out.append(rec.gather(p))
            if datum is not None:
                red.append(datum.gather(self.interior(p).contiguous()))
            self.v_step(st, p, 2, 1.0)
            self.surface(st)
        return torch.stack(out), torch.stack(red) if red else None

    def stage_a(self, st, res, rec, hist):
        w = self.kap.reshape(-1)[rec.idx] * self.dt * rec.coef
        for k in range(res.shape[0]):
            self.p_step(st, 3, -1.0)
            st[0].view(-1).index_add_(0, rec.idx.view(-1), -(w * res[k][:, None]).view(-1))
            p = self.p_sum(st)
            self.v_step(st, p, 3, -1.0)
            self.surface(st)
            if hist is not None:
                for f, x in enumerate((p, st[2], st[3])):
                    hist[k, f] = self.interior(x)

    def operator(self, res, rec, esource=False, datum=None, wavefield=None):
        """G G^T res, (nt, nr); stage A kept in windows of bounded size."""
        nt = res.shape[0]
        win = int(min(nt, max(1, 12e9 // (24 * self.n1 * self.n2))))
        starts = list(range(0, nt, win))
        hist = torch.empty(win, 3, self.n1, self.n2, dtype=_F64, device=self.dev)
        saved, st, cost = [], self.zeros(), 0.0
        for t0 in starts:
            saved.append([f.cpu() if len(starts) > 1 else f.clone() for f in st])
            self.stage_a(st, res[t0:t0 + win], rec, hist if t0 == starts[-1] else None)
        st, out, red = self.zeros(), [], []
        cut = 1 if esource else 0
        for t0, start in zip(reversed(starts), reversed(saved)):
            n = min(win, nt - t0)
            if t0 != starts[-1]:
                self.stage_a([f.to(self.dev) for f in start], res[t0:t0 + n], rec, hist)
            if esource:
                cost += sum(float((hist[k, 0] ** 2).sum()) for k in range(n)) * 0.5
            for k in range(n - 1, -1, -1):
                self.p_step(st, 3, 1.0)
                self.interior(st[0], cut).sub_(
                    self.dt * hist[k, 0][cut:self.n1 - cut, cut:self.n2 - cut]
                    * self.interior(self.kap, cut))
                p = self.p_sum(st)
                out.append(rec.gather(p))
                if datum is not None:
                    red.append(datum.gather(self.interior(p).contiguous()))
                if wavefield is not None:
                    wavefield.append(self.interior(p).cpu())
                self.v_step(st, p, 3, 1.0)
                b = self.interior(self.bu) if self.bu is not None else 1.0
                self.interior(st[2]).sub_(self.dt * hist[k, 1] * b)
                self.interior(st[3]).sub_(self.dt * hist[k, 2] * b)
                self.surface(st)
        return torch.stack(out), torch.stack(red) if red else None, cost

    def minres(self, b, rec, maxiter):
        """Paige and Saunders' MINRES on the time-reversed operator, shifted."""
        A = lambda x: self.operator(x, rec)[0].flip(0)  # noqa: E731
        shift = -MU * float(b.norm()) / float(self.operator(b, rec)[0].norm())
        x, w, w2 = (torch.zeros_like(b) for _ in range(3))
        r1 = r2 = b
        beta1 = beta = float(b.norm())
        oldb = dbar = eps = tnorm2 = 0.0
        cs, sn, phibar, y = -1.0, 0.0, beta1, b
        for itn in range(maxiter):
            v = y / beta
            y = A(v) - shift * v
            if itn:
                y = y - beta / oldb * r1
            alfa = float((v * y).sum())
            y = y - alfa / beta * r2
            r1, r2 = r2, y
            oldb, beta = beta, float(y.norm())
            tnorm2 += alfa ** 2 + oldb ** 2 + beta ** 2
            oldeps, delta = eps, cs * dbar + sn * alfa
            gbar, eps, dbar = sn * dbar - cs * alfa, sn * beta, -cs * beta
            gamma = math.hypot(gbar, beta)
            cs, sn = gbar / gamma, beta / gamma
            phi, phibar = cs * phibar, sn * phibar
            w1, w2 = w2, w
            w = (v - oldeps * w1 - delta * w2) / gamma
            x = x + phi * w
        return x, shift, phibar, math.sqrt(tnorm2)


def _filter(d, dt, band):
    """The band pass of filmartin2d (trapezoid with squared Hanning flanks)."""
    f = np.float32
    nt, nr = d.shape
    nto = 8
    while nto < nt:
        nto *= 2
    fe = f(1.0) / f(dt)
    flow, fhig, llow, lhig = (f(b) for b in band)
    if fhig > fe / f(2):
        fhig, lhig = fe / f(2), f(0)
    conv = f(int(f(nto) / fe))
    ilow, ihig, wlow, whig = (int(b * conv) + 1 for b in (flow, fhig, llow, lhig))
    if ilow - wlow < 1:
        wlow = ilow - 1
    if ihig + whig > nto:
        whig = nto - ihig
    han = lambda j, n: (0.5 * (math.cos(math.pi * (j - 1) / n) + 1.0) + 1e-6) ** 2  # noqa: E731
    w = np.zeros(nto + 1)
    for j in range(1, wlow + 1):
        w[ilow - j] = han(j, wlow)
    for j in range(1, whig + 1):
        w[ihig + j - 2] = han(j, whig)
    w[ilow - 1:ihig] = 1.0
    w += 1e-4
    x = torch.zeros(nto, nr, dtype=_F64, device=d.device)
    x[:nt] = d
    g = torch.from_numpy(w[:nto // 2 + 1].copy()).to(d.device)
    g[-1] = w[0]  # the packed transform keeps the last bin beside the first
    return torch.fft.irfft(torch.fft.rfft(x, dim=0) * g[:, None], n=nto, dim=0)[:nt]


def exact(case, seed):
    inp = _inputs(case, seed)
    if case["kind"] == "filter":
        return _filter(torch.from_numpy(inp["shots"][0]["data"].astype(np.float64)),
                       case["dt"], _band(case)).numpy()
    steps = case["nt"] * case["nshot"] * _sims(case)
    points = (case["n1"] + 2 * case["npml"]) * (case["n2"] + 2 * case["npml"])
    # seconds of the loops below: about 1 ms a step and 0.6 ns a point and step
    if steps * (1.0e-3 + 0.6e-9 * points) > 18.0 or not torch.cuda.is_available():
        return None
    wv = _Wave(case, inp)
    t64 = lambda a: torch.from_numpy(a.astype(np.float64)).to(wv.dev)  # noqa: E731
    host = lambda t: t.cpu().numpy()  # noqa: E731
    sh = inp["shots"][0]
    kind = case["kind"]
    if kind == "forward":
        out = [host(wv.forward(q["s"], wv.stations(q["src"]), wv.stations(q["rec"]))[0])
               for q in inp["shots"]]
        return out[0] if len(out) == 1 else out
    if kind == "ggt":
        return host(wv.operator(t64(sh["data"]), wv.stations(sh["rec"]))[0])
    if kind == "esource":
        wf = [] if case["wavefield"] else None
        sis, _, cost = wv.operator(t64(sh["data"]), wv.stations(sh["rec"]), True, wavefield=wf)
        return dict(sis=host(sis), cost=cost,
                    **({"wavefield": torch.stack(wf, -1).numpy()} if case["wavefield"] else {}))
    if kind == "minres":
        x, shift, rnorm, anorm = wv.minres(t64(sh["data"]), wv.stations(sh["rec"]),
                                           case["maxiter"])
        return dict(x=host(x), shift=shift, rnorm=rnorm, anorm=anorm)
    out = []
    datum = _Stations(inp["datum"], wv.h, wv.n1, wv.n2, 0, wv.dev)
    for q in inp["shots"]:
        rec = wv.stations(q["rec"])
        datar, red = wv.forward(q["s"], wv.stations(q["src"]), rec, datum)
        deltadr = (t64(q["data"]) - datar).flip(0)
        x = wv.minres(deltadr, rec, case["maxiter"])[0]
        esc, red2, _ = wv.operator(x, rec, True, datum)
        raw = red + red2
        r = dict(datar=datar, deltadr=deltadr, deltade=x, dataesc=esc, datae=datar + esc,
                 redatumed_raw=raw, redatumed=_filter(raw, case["dt"], _band(case)))
        out.append({k: host(v) for k, v in r.items()})
    return out
