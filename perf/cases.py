"""The work that users of this library have it do, as measurable cases.

A pass of a case is one stretch of a user's program between two looks at the results: so many
physical steps through the public entry points, then the state (and, where a program follows them,
the statistics or the inundation map) read back whole.  The sizes, boundary mixes and step counts
are those of the repository's configurations (`celeris_b200.cases`, C1-C5), of its tests and of its
benchmark; odd and ragged sizes stand beside the round ones.

`exact` is the same scheme in 64 bits in plain torch: reconstruction, central-upwind fluxes, the
Madsen-Sorensen terms, AB3 / AM4, the implicit solves (by parallel cyclic reduction) and the
boundaries, on the single-precision staggered bottom that the scheme defines its inputs on.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import celeris_b200 as cb
from celeris_b200 import cases

EULER, PREDICTOR, CORRECTOR = 0, 1, 2


def listed():
    return [
        # One displayed frame of an interactive program on the small flume: resetTimestep and
        # timestep for the predictor and for the corrector, then the texture to draw.  The smallest
        # call there is: latency and launches are all that counts.
        {"name": "frame_512x64", "kind": "flume", "api": "frame", "form": "mixed", "sizes": "512x64", "N": 1, "steps": 1},
        # The flume to its next log dump (logStep 100) in the plain form, the one that reproduces the
        # reference bit for bit and the default of `Engine`.
        {"name": "flume_plain_512x64", "kind": "flume", "api": "engine", "form": "plain", "sizes": "512x64", "N": 1, "steps": 100},
        # The plain form on a mid-size closed basin of odd sides.
        {"name": "basin_plain_1001x777", "kind": "cone", "api": "engine", "form": "plain", "sizes": "1001x777", "N": 1, "steps": 20},
        # The same flume as a batch of one with graphs, in the compensated form; its inundation map too.
        {"name": "flume_512x64", "kind": "flume", "api": "batch", "form": "mixed", "sizes": "512x64", "N": 1, "steps": 200, "aux": True},
        # A short parameter study followed step by step: time steps up, statistics down, every step.
        {"name": "monitor_8x256", "kind": "ensemble", "api": "monitor", "form": "mixed",
         "sizes": "256x256,256x256,512x256,256x256,128x96,512x256,256x256,161x131", "N": 1, "steps": 50},
        # Solitary wave running up a cone in a closed basin, one domain.
        {"name": "cone_1024x1024", "kind": "cone", "api": "batch", "form": "mixed", "sizes": "1024x1024", "N": 1, "steps": 200},
        # Harbour: recorded water levels on two sides, a wide wall on the third, ragged sides, two correctors.
        {"name": "harbour_1017x643", "kind": "harbour", "api": "engine", "form": "mixed", "sizes": "1017x643", "N": 2, "steps": 50},
        # An open coast under an irregular sea: spectrum wave-maker, three sponges, friction, breaking.
        {"name": "coast_2048x2048", "kind": "coast", "api": "batch", "form": "mixed", "sizes": "2048x2048", "N": 1, "steps": 60, "waves": 64},
        # Many small domains with friction in one batch, default tuning.
        {"name": "ensemble_small_40", "kind": "ensemble", "api": "batch", "form": "mixed",
         "sizes": ",".join("%dx%d" % (128 + 32 * (7 * k % 13), 128 + 32 * (5 * k % 13)) for k in range(40)),
         "N": 1, "steps": 150, "manning": 0.02},
        # Adaptive time steps chosen on the device, ragged members.
        {"name": "ensemble_adaptive_12", "kind": "ensemble", "api": "batch", "form": "mixed",
         "sizes": "256x256,512x256,1024x512,300x1021,512x256,799x601,1024x512,256x256,1024x1024,512x256,333x255,1024x512",
         "N": 1, "steps": 100, "adaptive": True},
        # Single precision without compensation and without a corrector (the cheapest run there is).
        {"name": "ensemble_fp32_ab3_12", "kind": "ensemble", "api": "batch", "form": "fused",
         "sizes": "1024x1024,512x256,2048x512,256x256,1024x512,777x613,512x256,1024x1024,2048x512,256x256,450x1100,1024x512",
         "N": 0, "steps": 100, "stencil": 96},
        # The uneven ensemble of the benchmark (its five member sizes), on the stencil that its tuner picks.
        {"name": "ensemble_uneven_28", "kind": "ensemble", "api": "batch", "form": "mixed",
         "sizes": ",".join(("256x256", "512x256", "1024x512", "1024x1024", "2048x512")[(k * k + k // 3) % 5] for k in range(28)),
         "N": 1, "steps": 200, "stencil": 96, "stats": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flume", "cone", "harbour", "coast", "ensemble", "ensemble", "ensemble"])
    if kind == "ensemble":
        n = _log_int(rng, 2, 40)
        api = rng.choice(["batch", "batch", "monitor"])
        N = rng.choice([0, 1, 1, 2])
        side = 420 if api == "monitor" else 1500
        sizes, cells = [], 0
        for _ in range(n):
            nx, ny = _log_int(rng, 96, side), _log_int(rng, 96, side)
            if cells + nx * ny > 8_000_000:
                break
            sizes.append("%dx%d" % (nx, ny))
            cells += nx * ny
        c = {"kind": kind, "api": api, "form": rng.choice(["mixed", "mixed", "fused"]), "sizes": ",".join(sizes), "N": N,
             "steps": _log_int(rng, 20, 60 if api == "monitor" else 120)}
        if rng.random() < 0.3 and api == "batch":
            c["adaptive"] = True
        if rng.random() < 0.4:
            c["manning"] = 0.02
        if rng.random() < 0.5:
            c["stencil"] = rng.choice([96, 128])
        return c
    if kind == "flume":
        api, form = rng.choice([("frame", "mixed"), ("frame", "fused"), ("engine", "plain"), ("batch", "mixed"), ("batch", "fused")])
        return {"kind": kind, "api": api, "form": form, "sizes": "%dx%d" % (_log_int(rng, 500, 900), _log_int(rng, 33, 200)),
                "N": 1, "steps": 1 if api == "frame" else _log_int(rng, 30, 120)}
    if kind == "cone":
        api, form = rng.choice([("batch", "mixed"), ("engine", "mixed"), ("engine", "plain"), ("batch", "fused")])
        side = 1100 if form == "plain" else 1800
        return {"kind": kind, "api": api, "form": form, "sizes": "%dx%d" % (_log_int(rng, 200, side), _log_int(rng, 200, side)),
                "N": rng.choice([1, 1, 2]), "steps": _log_int(rng, 10, 20) if form == "plain" else _log_int(rng, 30, 120)}
    api, form = rng.choice([("batch", "mixed"), ("engine", "mixed"), ("batch", "fused")])
    c = {"kind": kind, "api": api, "form": form, "sizes": "%dx%d" % (_log_int(rng, 300, 1900), _log_int(rng, 200, 1900)),
         "N": rng.choice([1, 1, 2]), "steps": _log_int(rng, 20, 60)}
    if kind == "coast":
        c["waves"] = _log_int(rng, 8, 90)
    return c


# ---- inputs -----------------------------------------------------------------------------------

def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]


def _sea(p, bottom, rng):
    """A hot start: a few progressive waves over the still water, fading out toward the shore."""
    ny, nx = bottom.shape
    dx, dy = p.width / (p.nx - 1), p.length / (p.ny - 1)
    x, y = np.arange(nx)[None, :] * dx, np.arange(ny)[:, None] * dy
    depth = np.maximum(0.0, -bottom)
    deep = max(0.3, float(depth.max()))
    eta, hu, hv = np.zeros(bottom.shape), np.zeros(bottom.shape), np.zeros(bottom.shape)
    for _ in range(4):
        th, k = rng.uniform(-0.5, 0.5), 2 * math.pi / (deep * rng.uniform(6, 14))
        e = 0.005 * deep * rng.uniform(0.5, 1.5) * np.cos(k * (math.cos(th) * x + math.sin(th) * y) + rng.uniform(0, 6.28))
        c = math.sqrt(9.81 * deep)
        eta, hu, hv = eta + e, hu + c * math.cos(th) * e, hv + c * math.sin(th) * e
    fade = np.clip(depth / (0.3 * deep), 0.0, 1.0) ** 2
    s = np.zeros(bottom.shape + (4,), np.float32)
    s[..., 0], s[..., 1], s[..., 2] = np.maximum(fade * eta, bottom), fade * hu, fade * hv
    return s


def _uts_table(rng):
    """A recorded signal: rows of (t, eta, hu, hv)."""
    t = np.linspace(0.0, 400.0, 801)
    per = rng.uniform(6.0, 12.0)
    e = 0.1 * np.sin(2 * np.pi * t / per) + 0.03 * np.sin(4 * np.pi * t / per + rng.uniform(0, 6.28))
    return np.stack([t, e, 3.0 * e, 0.2 * e], axis=1)


def _bottom(p, z):
    """The staggered bottom as the scheme defines it, in single precision: the grid sampled at the
    cell corners, BA / BX / BY the means of a cell's four corners and of its east and north pairs."""
    f = np.float32
    ny, nx = z.shape
    W, L = f(p.width), f(p.length)
    x = (np.arange(p.nx + 5, dtype=f) - f(2.5)) / f(p.nx - 1) * W - W / f(2)
    y = (np.arange(p.ny + 5, dtype=f) - f(2.5)) / f(p.ny - 1) * L
    x = np.clip((x + W / f(2)) / W * f(nx - 1), f(0), f(nx - 1))
    y = np.clip(y / L * f(ny - 1), f(0), f(ny - 1))
    x0, x1, y0, y1 = (g(v).astype(int) for v in (x, y) for g in (np.floor, np.ceil))
    fx, fy = (x - x0.astype(f))[None, :], (y - y0.astype(f))[:, None]
    lo, hi = (z[r][:, x0] + fx * (z[r][:, x1] - z[r][:, x0]) for r in (y0, y1))
    c = lo + fy * (hi - lo)
    q, h = f(0.25), f(0.5)
    z00, z10, z01, z11 = c[:-1, :-1], c[:-1, 1:], c[1:, :-1], c[1:, 1:]
    return ((q * z00 + q * z10) + q * z01) + q * z11, h * z10 + h * z11, h * z01 + h * z11


def _members(case, seed):
    """[(params, bathymetry, hot start or None, (uts table or None, its buffers))] of a case."""
    out = []
    for k, (nx, ny) in enumerate(_sizes(case)):
        rng = np.random.default_rng([int(seed), k])
        keep = (None, [])
        if case["kind"] == "flume":
            p, z, _, _ = cases.config1(nx, ny, correction_steps=case["N"])
        elif case["kind"] == "cone":
            p, z, _, _ = cases.config3(nx, ny, correction_steps=case["N"])
            p.length = p.width / (nx - 1) * (ny - 1)   # square cells
            z = cases.config3(nx, nx)[1]
            z = z[(nx - ny) // 2:(nx - ny) // 2 + ny] if ny <= nx else np.pad(z, (((ny - nx) // 2, ny - nx - (ny - nx) // 2), (0, 0)), mode="edge")
            s = p.solitons[0]
            s.H, s.theta, s.xc, s.yc = rng.uniform(0.02, 0.035), rng.uniform(-0.2, 0.2), rng.uniform(2.0, 5.0), 0.5 * p.length
        elif case["kind"] == "coast":
            p, z, _, _ = cases.config2(nx, ny, n_waves=case["waves"], member=int(seed) % 1_000_003, correction_steps=case["N"])
            z = np.minimum(z, 3.0)
        else:
            p, z, _, _ = cases.ensemble_member(nx, ny, rng, case["N"], manning=case.get("manning", 0.0))
            z = np.minimum(z, 5.0)
            if case["kind"] == "harbour":
                table = _uts_table(rng)
                for side, kind, width in ((p.west, 4, 2), (p.north, 4, 2), (p.east, 0, 3), (p.south, 0, 2)):
                    side.type, side.width = kind, width
                keep = (table, cases.attach_uts(p, "west", table) + cases.attach_uts(p, "north", table))
            if case["N"] == 0:
                p.timestep *= 0.5   # pure AB3 is stable to half the Courant number
        p.adaptive = int(bool(case.get("adaptive")))
        z = np.ascontiguousarray(z, dtype=np.float32)
        hot = None if case["kind"] == "cone" else _sea(p, _bottom(p, z)[0].astype(np.float64), rng)
        out.append((p, z, hot, keep))
    return out


def prepare(case, seed):
    ms = _members(case, seed)
    if case["api"] in ("engine", "frame"):
        p, z, hot, keep = ms[0]
        sim = cb.Engine(p, z, case["form"])
        if hot is not None:
            sim.set_state(hot)
    else:
        sim = cb.Batch([(p, z) for p, z, _, _ in ms], case["form"])
        if "stencil" in case:
            sim.set_stencil_rows(2)
            sim.set_stencil_width(case["stencil"])
        sim.use_graph(True)
        for i, (_, _, hot, _) in enumerate(ms):
            if hot is not None:
                sim.set_state(i, hot)
    dt = np.array([p.timestep for p, _, _, _ in ms], dtype=np.float32)
    return {"case": case, "sim": sim, "keep": [m[3] for m in ms], "dt": dt}


def _table(stats):
    # the per-cell terms are single precision, and a program logs their totals so
    return np.array([[s[k] for k in ("mass", "kinetic_energy", "potential_energy", "max_speed", "max_depth", "cfl_rate",
                                     "timestep", "total_time", "mass_full")] for s in stats], dtype=np.float32)


def run(state):
    case, sim = state["case"], state["sim"]
    if case["api"] == "frame":
        for _ in range(case["steps"]):
            for _ in range(1 + case["N"]):
                s = sim.reset_timestep()
                sim.timestep()
        return {"stats": _table([s]), "state": [sim.state()]}
    if case["api"] == "engine":
        sim.physical_steps(case["steps"])
        return {"state": [sim.state()]}
    out = {}
    if case["api"] == "monitor":
        rows = []
        for _ in range(case["steps"]):
            sim.set_timestep(state["dt"])
            sim.step(1)
            rows.append(_table(sim.stats()))
        out["stats"] = np.stack(rows)
    else:
        sim.step(case["steps"])
        if case.get("stats"):
            out["stats"] = _table(sim.stats())
    out["state"] = [sim.state(i) for i in range(sim.n)]
    if case.get("aux"):
        out["aux"] = [sim.aux(i) for i in range(sim.n)]
    return out


def work(case):
    """Per cell and pass of a step: the state in and out (12 + 12 bytes), the bottom (4), the implicit
    systems (two coefficients a direction, 16), the derivatives of this pass out (20) and those it
    combines with in (two older levels, 40; in a corrector their sum, 20), the inundation and breaking
    record in and out (16); the compensated form the low words of the state in and out (24), a
    corrector the state it corrects (12).  Read back: 16 bytes a texel (the inundation map as much).
    Operations: about 400 a cell and pass."""
    cells = sum(nx * ny for nx, ny in _sizes(case))
    texels = sum((nx + 4) * (ny + 4) for nx, ny in _sizes(case))
    comp = 24 if case["form"] == "mixed" else 0
    per_step = (120 + comp) + case["N"] * (112 + comp)
    back = 16 * texels * (2 if case.get("aux") else 1)
    return {"bytes": float(cells * per_step * case["steps"] + back), "flops": 400.0 * cells * (1 + case["N"]) * case["steps"]}


# ---- the scheme in 64 bits ----------------------------------------------------------------------

def _sh(a, dx, dy):
    """a at (x + dx, y + dy); what wraps round at the rim is never used."""
    return torch.roll(a, (-dy, -dx), (0, 1))


def _minmod(z1, z2, z3):
    mn, mx = torch.minimum(torch.minimum(z1, z2), z3), torch.maximum(torch.maximum(z1, z2), z3)
    return torch.where(mn > 0, mn, torch.where(mx < 0, mx, torch.zeros_like(mn)))


class _Exact:
    def __init__(self, p, z, hot, table):
        self.p, self.table = p, table
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.BA, self.BX, self.BY = (torch.tensor(b.astype(np.float64), device=self.dev) for b in _bottom(p, z))
        self.nx, self.ny, self.NX, self.NY = p.nx, p.ny, p.nx + 4, p.ny + 4
        self.dx, self.dy = p.width / (p.nx - 1), p.length / (p.ny - 1)
        self.g, self.sl = p.gravity, p.still_water_elevation
        self.eps = min(p.epsilon, max(self.dx, self.dy) ** 4)
        self.I = (slice(2, self.NY - 2), slice(2, self.NX - 2))
        d = torch.clamp(self.sl - self.BA, min=0.0)
        self.d = d
        self.ddx = (-_sh(d, 2, 0) + 8 * _sh(d, 1, 0) - 8 * _sh(d, -1, 0) + _sh(d, -2, 0)) / (12 * self.dx)
        self.ddy = (-_sh(d, 0, 2) + 8 * _sh(d, 0, 1) - 8 * _sh(d, 0, -1) + _sh(d, 0, -2)) / (12 * self.dy)
        self.sys = [self._factor(self.dx, self.ddx, 1), self._factor(self.dy, self.ddy, 0)]
        S = torch.zeros((3, self.NY, self.NX), dtype=torch.float64, device=self.dev)
        if hot is not None:
            S = torch.tensor(hot[..., :3].astype(np.float64), device=self.dev).permute(2, 0, 1).contiguous()
        else:
            y = torch.arange(self.NY, dtype=torch.float64, device=self.dev).clamp(2, self.ny + 1).long()
            x = torch.arange(self.NX, dtype=torch.float64, device=self.dev).clamp(2, self.nx + 1).long()
            B = self.BA[y][:, x]
            S[0] = torch.clamp(B, min=self.sl)
            X = torch.arange(self.NX, dtype=torch.float64, device=self.dev)[None, :] * self.dx
            Y = torch.arange(self.NY, dtype=torch.float64, device=self.dev)[:, None] * self.dy
            for q in range(p.n_solitons):
                s = p.solitons[q]
                dep = torch.clamp(self.sl - B, min=0.0)
                wet = dep > 0
                dep = torch.where(wet, dep, torch.ones_like(dep))
                K = torch.sqrt(0.75 * abs(s.H) / dep ** 3)
                ch = torch.cosh(K * ((X - s.xc) * math.cos(s.theta) + (Y - s.yc) * math.sin(s.theta)))
                e = torch.where(wet, s.H / (ch * ch), torch.zeros_like(dep))
                c = torch.sqrt(self.g * (s.H + dep))
                S += torch.stack([e, c * math.cos(s.theta) * e, c * math.sin(s.theta) * e])
        self.S = S

    def _factor(self, h, dd, axis):
        """The implicit system along an axis as the multipliers of parallel cyclic reduction."""
        d = self.d if self.p.boussinesq else torch.zeros_like(self.d)
        dd = dd if self.p.boussinesq else torch.zeros_like(dd)
        K1, K2 = (1 / 15 + 1 / 3) * d * d / (h * h), d * dd / (6 * h)   # (d / h^2) (...) / 72
        a, b, c = (t[self.I].clone() for t in (-K1 + K2, 1 + 2 * K1, -(K1 + K2)))
        n = a.shape[axis]
        a.narrow(axis, 0, 1).zero_()
        c.narrow(axis, n - 1, 1).zero_()

        def at(t, s, fill):   # t at i + s along the axis
            o = torch.full_like(t, fill)
            if s > 0:
                o.narrow(axis, 0, n - s).copy_(t.narrow(axis, s, n - s))
            else:
                o.narrow(axis, -s, n + s).copy_(t.narrow(axis, 0, n + s))
            return o

        levels, s = [], 1
        while s < n:
            k1, k2 = a / at(b, -s, 1.0), c / at(b, s, 1.0)
            a, b, c = -at(a, -s, 0.0) * k1, b - at(c, -s, 0.0) * k1 - at(a, s, 0.0) * k2, -at(c, s, 0.0) * k2
            levels.append((s, k1, k2))
            s *= 2
        return axis, levels, b

    @staticmethod
    def _solve(system, r):
        axis, levels, b = system
        n = r.shape[axis]
        for s, k1, k2 in levels:
            o = r.clone()
            o.narrow(axis, s, n - s).sub_(k1.narrow(axis, s, n - s) * r.narrow(axis, 0, n - s))
            o.narrow(axis, 0, n - s).sub_(k2.narrow(axis, 0, n - s) * r.narrow(axis, s, n - s))
            r = o
        return r / b

    def _by_h(self, h):
        h4 = h ** 4
        return math.sqrt(2.0) * h / torch.sqrt(h4 + torch.clamp(h4, min=self.eps))

    def _faces(self, dx, dy, Bm, Bp):
        """Depth, velocities and level on a cell's two faces along an axis."""
        tt = 2 * self.p.theta
        lo, hi = [], []
        for q in range(3):
            c, w, e = self.S[q], _sh(self.S[q], -dx, -dy), _sh(self.S[q], dx, dy)
            g2 = 0.25 * _minmod(tt * (c - w), e - w, tt * (e - c))
            lo.append(c - g2)
            hi.append(c + g2)
        ww, we, c = lo[0], hi[0], self.S[0]
        c1 = we < Bp
        c2 = ~c1 & (ww < Bm)
        nwe = torch.where(c1, Bp, torch.where(c2, torch.maximum(Bp, 2 * c - Bm), we))
        nww = torch.where(c1, torch.maximum(Bm, 2 * c - Bp), torch.where(c2, Bm, ww))
        out = []
        for w, B, v in ((nww, Bm, lo), (nwe, Bp, hi)):
            h = w - B
            q = self._by_h(h)
            out.append((h, q * v[1], q * v[2]))
        return out

    def _flux(self, minus, plus, n):
        """Central-upwind flux between a face's two sides; n: the normal velocity's index."""
        hm, hp, g = minus[0], plus[0], self.g
        cm, cp = torch.sqrt(g * hm), torch.sqrt(g * hp)
        ap = torch.clamp(torch.maximum(minus[n] + cm, plus[n] + cp), min=0.0)
        am = torch.clamp(torch.minimum(minus[n] - cm, plus[n] - cp), max=0.0)
        den = ap - am
        live = den != 0
        den = torch.where(live, den, torch.ones_like(den))
        out = []
        for k in range(3):
            Um, Up = (hm, hp) if k == 0 else (hm * minus[k], hp * plus[k])
            Fm, Fp = Um * minus[n], Up * plus[n]
            if k == n:
                Fm, Fp = Fm + 0.5 * g * hm * hm, Fp + 0.5 * g * hp * hp
            out.append(torch.where(live, (ap * Fm - am * Fp + ap * am * (Up - Um)) / den, torch.zeros_like(den)))
        return out

    def _rates(self):
        """The derivatives (w, hu, hv) and the mixed dispersion terms F*, G* of the state."""
        S, dx, dy, d, ddx, ddy = self.S, self.dx, self.dy, self.d, self.ddx, self.ddy
        west, east = self._faces(1, 0, _sh(self.BX, -1, 0), self.BX)
        south, north = self._faces(0, 1, _sh(self.BY, 0, -1), self.BY)
        xf = self._flux(east, [_sh(v, 1, 0) for v in west], 1)
        yf = self._flux(north, [_sh(v, 0, 1) for v in south], 2)
        f = [(_sh(xf[k], -1, 0) - xf[k]) / dx + (_sh(yf[k], 0, -1) - yf[k]) / dy for k in range(3)]
        e = S[0] - self.sl
        r, l, u, b = _sh(e, 1, 0), _sh(e, -1, 0), _sh(e, 0, 1), _sh(e, 0, -1)
        ur, ul, br, bl = _sh(e, 1, 1), _sh(e, -1, 1), _sh(e, 1, -1), _sh(e, -1, -1)
        exx, eyy, exy = (r - 2 * e + l) / dx ** 2, (u - 2 * e + b) / dy ** 2, 0.25 * (ur - br - ul + bl) / (dx * dy)
        exxx = (_sh(e, 2, 0) - 2 * r + 2 * l - _sh(e, -2, 0)) / (2 * dx ** 3)
        eyyy = (_sh(e, 0, 2) - 2 * u + 2 * b - _sh(e, 0, -2)) / (2 * dy ** 3)
        exyy = (ur - ul - 2 * r + 2 * l + br - bl) / (2 * dx * dy ** 2)
        exxy = (ur + ul - 2 * u + 2 * b - br - bl) / (2 * dy * dx ** 2)
        Bg = self.g / 15
        px = Bg * d ** 3 * (exxx + exyy) + Bg * d ** 2 * (ddx * (2 * exx + eyy) + ddy * exy)
        py = Bg * d ** 3 * (eyyy + exxy) + Bg * d ** 2 * (ddy * (exx + 2 * eyy) + ddx * exy)
        h = torch.clamp(S[0] - self.BA, min=0.0)
        fr = torch.zeros_like(h)
        if self.p.friction != 0:
            q = self._by_h(h)
            k = self.g * self.p.friction ** 2 * q.abs() ** 0.3333 if self.p.manning else self.p.friction
            fr = k * torch.sqrt(S[1] ** 2 + S[2] ** 2) * q * q
        f[1] = f[1] - self.g * h * (self.BX - _sh(self.BX, -1, 0)) / dx - S[1] * fr + px
        f[2] = f[2] - self.g * h * (self.BY - _sh(self.BY, 0, -1)) / dy - S[2] * fr + py
        cross = [d / 6 * (ddx * (_sh(v, 0, 1) - _sh(v, 0, -1)) / (2 * dy) + ddy * (_sh(v, 1, 0) - _sh(v, -1, 0)) / (2 * dx))
                 for v in (S[2], S[1])]
        return torch.stack([t[self.I] for t in f + cross])

    def _wave(self, x, y, t, dep, amp, per, th, phase):
        om = 2 * math.pi / per
        wet = dep > 1e-4
        dep = torch.where(wet, dep, torch.ones_like(dep))
        k = om * om / (self.g * torch.sqrt(torch.tanh(om * om * dep / self.g)))
        e = amp * torch.sin(om * t - math.cos(th) * x * k - math.sin(th) * y * k + phase)
        e = torch.where(wet, e, torch.zeros_like(e))
        return e, om / k * math.cos(th) * e, om / k * math.sin(th) * e

    def _side(self, side, b, t, dt):
        NX, NY = self.NX, self.NY
        x0, x1, y0, y1 = {"east": (NX - b.width, NX, 0, NY), "west": (0, b.width, 0, NY),
                          "north": (0, NX, NY - b.width, NY), "south": (0, NX, 0, b.width)}[side]
        x0, y0, x1, y1 = max(x0, 0), max(y0, 0), min(x1, NX), min(y1, NY)
        X = torch.arange(x0, x1, dtype=torch.float64, device=self.dev)[None, :].expand(y1 - y0, -1)
        Y = torch.arange(y0, y1, dtype=torch.float64, device=self.dev)[:, None].expand(-1, x1 - x0)
        at = (slice(y0, y1), slice(x0, x1))
        along_x = side in ("east", "west")
        out = torch.zeros((3, y1 - y0, x1 - x0), dtype=torch.float64, device=self.dev)
        if b.type == 0:      # wall: the mirrored texel (coordinates truncate toward zero), zero outside
            m = {"west": 4, "south": 4, "east": 2 * self.nx + 2, "north": 2 * self.ny + 2}[side]
            qx = torch.trunc(m - (X + 0.5)).long() if along_x else X.long()
            qy = Y.long() if along_x else torch.trunc(m - (Y + 0.5)).long()
            ok = (qx >= 0) & (qx < NX) & (qy >= 0) & (qy < NY)
            v = self.S[:, qy.clamp(0, NY - 1), qx.clamp(0, NX - 1)]
            out = torch.where(ok, v, torch.zeros_like(v))
            out[1 if along_x else 2] *= -1
        elif b.type == 1:    # sponge
            dist = {"west": X * self.dx, "east": (NX - X) * self.dx, "south": Y * self.dy, "north": (NY - Y) * self.dy}[side]
            L = b.width * (self.dx if along_x else self.dy)
            fn = lambda v: torch.sin(0.5 * math.pi * torch.clamp(v / L, max=1.0)) ** 2  # noqa: E731
            gam = fn(dist) / fn(dist + torch.sqrt(self.g * torch.clamp(b.sea_level - self.BA[at], min=1e-4)) * dt)
            out = gam * self.S[(slice(None),) + at]
            out[0] += (1 - gam) * b.sea_level
        elif b.type == 4:    # recorded levels
            out += torch.tensor([np.interp(t, self.table[:, 0], self.table[:, q]) for q in (1, 2, 3)],
                                dtype=torch.float64, device=self.dev)[:, None, None]
            out[0] += b.sea_level
        else:                # wave-makers
            dep = torch.clamp(b.sea_level - self.BA[at], min=0.0)
            x, y = (X - NX if side == "east" else X) * self.dx, (Y - NY if side == "north" else Y) * self.dy
            if b.type == 2:
                waves = [(b.amplitude, b.period, b.theta, 0.0)]
            else:
                waves = [tuple(b.waves[i]) for i in range(b.n_waves)]
            for wv in waves:
                out += torch.stack(self._wave(x, y, t, dep, *wv))
            out[0] += b.sea_level
            if b.type == 3:  # only the texels along the interior
                n, v = (self.ny, Y) if along_x else (self.nx, X)
                out *= ((v >= 2) & (v < n + 2)).to(torch.float64)
        self.S[(slice(None),) + at] = out

    def _cfl(self):
        i = (slice(2, 2 + 4 * (self.ny // 4)), slice(2, 2 + 4 * (self.nx // 4)))
        h = torch.clamp(self.S[0][i] - self.BA[i], min=0.0)
        q, c = self._by_h(h), torch.sqrt(self.g * h)
        return max(float(((q * self.S[1][i]).abs() + c).max()) / self.dx, float(((q * self.S[2][i]).abs() + c).max()) / self.dy)

    def run(self, steps):
        p = self.p
        base = float(np.float32(p.timestep))
        t, old, oldold, dts, target = 0.0, None, None, [base, base], None
        for step in range(steps):
            cur, pred = self.S, None
            kinds = [EULER] if step < 2 else [PREDICTOR] + [CORRECTOR] * p.correction_steps
            if target is None and p.adaptive:
                target = base * self._cfl()
            for kind in kinds:
                dt = base
                f = self._rates()
                if kind == EULER:
                    inc = dt * f[:3]
                elif kind == PREDICTOR and p.adaptive:
                    want = max(target / self._cfl(), base * p.min_timestep_ratio)
                    dt = p.ema_alpha * want + (1 - p.ema_alpha) * dts[0] if want > dts[0] else want
                    A, K = self._ab3(dt, *dts)
                    inc = dt / 6 * (A[0] * f[:3] + A[1] * old[:3] + A[2] * oldold[:3])
                    inc[1:] += K[0] * f[3:] + K[1] * old[3:] + K[2] * oldold[3:]
                elif kind == PREDICTOR:
                    inc = dt / 12 * (23 * f[:3] - 16 * old[:3] + 5 * oldold[:3])
                    inc[1:] += 2 * f[3:] - 3 * old[3:] + oldold[3:]
                else:
                    inc = dt / 24 * (9 * f[:3] + 19 * pred[:3] - 5 * old[:3] + oldold[:3])
                    inc[1:] += f[3:] - pred[3:]
                if kind == PREDICTOR:
                    pred = f
                S = torch.zeros_like(cur)
                S[0][self.I] = cur[0][self.I] + inc[0]
                S[1][self.I] = cur[1][self.I] + self._solve(self.sys[0], inc[1])
                S[2][self.I] = cur[2][self.I] + self._solve(self.sys[1], inc[2])
                self.S = S
                for side in ("east", "north", "west", "south"):
                    self._side(side, getattr(p, side), t, dt)
            old, oldold = f, old if old is not None else torch.zeros_like(f)
            t, dts = t + dt, [dt, dts[0]]
        out = torch.zeros((self.NY, self.NX, 4), dtype=torch.float64, device=self.dev)
        out[..., :3] = self.S.permute(1, 2, 0)
        return out.cpu()

    @staticmethod
    def _ab3(dt, d1, d2):
        """Variable-step third-order Adams-Bashforth weights and, folded with them, those of the time
        derivative of F*, G* (differences over the last three levels)."""
        s = d1 + d2
        A = [dt / d1 * (2 * dt + 6 * d1 + 3 * d2) / s + 6, -dt / d1 * (2 * dt + 3 * d1 + 3 * d2) / d2, dt / d2 * (2 * dt + 3 * d1) / s]
        D = [[(2 * d1 + d2) / (d1 * s), -s / (d1 * d2), d1 / (d2 * s)],
             [d2 / (d1 * s), (d1 - d2) / (d1 * d2), -d1 / (d2 * s)],
             [-d2 / (d1 * s), s / (d1 * d2), -(d1 + 2 * d2) / (d2 * s)]]
        return A, [dt / 6 * sum(A[m] * D[m][j] for m in range(3)) for j in range(3)]


def exact(case, seed):
    """The states in 64 bits; members beyond what about 20 seconds compute have none, nor have the
    statistics and the inundation map."""
    budget = 6e8 if torch.cuda.is_available() else 2e7   # cell-passes
    states = []
    for (p, z, hot, keep), (nx, ny) in zip(_members(case, seed), _sizes(case)):
        cost = (nx * ny + 150_000) * (1 + case["N"]) * case["steps"]
        if cost > budget:
            states.append(None)
            continue
        budget -= cost
        # a frame counts passes, and the first two passes of a run are Euler steps of their own
        states.append(_Exact(p, z, hot, keep[0]).run(case["steps"] + (1 if case["api"] == "frame" else 0)))
    out = {"state": states}
    if case["api"] in ("frame", "monitor") or case.get("stats"):
        out["stats"] = None
    if case.get("aux"):
        out["aux"] = [None] * len(states)
    return out
