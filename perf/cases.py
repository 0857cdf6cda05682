"""Performance cases: simulations a user of sph_gb300 runs, each through the public entry points.

One pass advances a scene (``Scene.step``) or a pool of scenes (``Pool.step``) by a few time steps and reads the
fluid's state back, as a program that renders or stores frames does.  The scene keeps evolving from pass to pass,
as it does in a running simulation.  Kinds of cases:

* ``wcsph``  a block settling in a box: a cube boundary with XSPH viscosity, or Akinci walls with fluid and boundary
             XSPH; 8,000 particles in the unit cube is the repository's CPU-runnable configuration (there in FP64);
* ``dam``    DFSPH dam break with Akinci walls in a 1.5 x 0.8 x 0.8 m box (125,000 particles at r = 5 mm), optionally
             with XSPH, surface tension, adhesion and a sphere obstacle;
* ``drop``   PCISPH drop onto a pool: standard viscosity, surface tension, adhesion (81k and 490k particles);
* ``mix``    a pool of independent DFSPH scenes of 2k-64k particles with obstacles, advanced together.

Lattices are jittered and thrown with a seeded velocity: an undisturbed lattice holds many pairs at exactly the
support radius, where rounding alone decides whether they count.  The FP32 form's state holds FP32 values (the
library hands them out in float64 arrays), so its outputs are returned as float32; the FP64 form's as float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import sph_gb300
from sph_gb300 import workloads

DFSPH, WCSPH, PCISPH = 2, 0, 1
MIX_CAP = 256  # the benchmark's mix


def _wcsph(name, n, precision, boundary, steps, graph=True):
    return dict(name=name, kind="wcsph", n=n, precision=precision, boundary=boundary, steps=steps, graph=graph)


def _dam(name, n, precision, forces, steps, graph=True):
    return dict(name=name, kind="dam", n=n, precision=precision, forces=forces, steps=steps, graph=graph)


def _drop(name, radius, precision, steps):
    return dict(name=name, kind="drop", radius=radius, precision=precision, steps=steps, graph=True)


def _mix(name, scenes, steps):
    return dict(name=name, kind="mix", scenes=scenes, precision="f32", steps=steps, graph=True)


def listed():
    return [
        # the smallest call: one step of the smallest scene of the mix, launched kernel by kernel (the default mode)
        _dam("dfsph_2k_one_step", 2000, "f32", False, 1, graph=False),
        # the repository's first configuration, in the reference's own precision and in the production form
        _wcsph("wcsph_8k_f64", 8000, "f64", "cube", 20),
        _wcsph("wcsph_8k", 8000, "f32", "cube", 50),
        # WCSPH at an ordinary size, walls sampled as particles, a ragged block
        _wcsph("wcsph_90k_akinci", 90011, "f32", "akinci", 20),
        # the scene sizes of the batched mix, run alone
        _dam("dfsph_13k", 13001, "f32", False, 10),
        # every non-pressure force at once, around an obstacle
        _dam("dfsph_50k_forces", 50000, "f32", True, 5),
        # the repository's second configuration, in both precisions
        _dam("dfsph_125k", 125000, "f32", False, 20),
        _dam("dfsph_125k_f64", 125000, "f64", False, 5),
        # the repository's third configuration at its two sizes
        _drop("pcisph_drop_81k", 0.005, "f32", 10),
        _drop("pcisph_drop_490k", 0.00275, "f32", 5),
        # the repository's fourth configuration (the benchmark's headline), and a smaller batch
        _mix("mix_24", 24, 20),
        _mix("mix_256", MIX_CAP, 20),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["wcsph", "wcsph", "dam", "dam", "dam", "drop", "mix"])
    if kind == "wcsph":
        precision = rng.choice(["f32", "f32", "f64"])
        n = size(1000, 125000 if precision == "f32" else 20000)
        c = _wcsph("", n, precision, rng.choice(["cube", "akinci"]), 10 if n < 40000 else 5)
    elif kind == "dam":
        precision = rng.choice(["f32", "f32", "f32", "f64"])
        n = size(1000, 500000 if precision == "f32" else 100000)
        c = _dam("", n, precision, rng.random() < 0.35, 5)
    elif kind == "drop":
        c = _drop("", round(math.exp(rng.uniform(math.log(0.00275), math.log(0.011))), 5), "f32", 5)
    else:
        c = _mix("", size(4, MIX_CAP), rng.choice([5, 10]))
    del c["name"]
    return c


# ---- scenes --------------------------------------------------------------------------------------------------------

def _ragged(n):
    """Block dimensions whose product is about n."""
    a = max(2, int(round(n ** (1.0 / 3.0))))
    b = max(2, int(round(math.sqrt(n / a))))
    return a, b, max(2, int(round(n / (a * b))))


def _block(r, corner, dims):
    mn = np.asarray(corner, dtype=np.float64)
    return sph_gb300.fluid_block(r, mn, mn + 2.0 * r * np.asarray(dims) + 1e-9)


def _geometry(case):
    """[(fluid points, boundary points or None, parameters)]: the lattices and walls, the same for every seed."""
    kind = case["kind"]
    if kind == "wcsph":
        dims = _ragged(case["n"])
        p = dict(method=WCSPH, stiffness=1000.0, gamma=7.0, dt=1e-4, visc_method=2, visc=0.01)
        if case["boundary"] == "cube":
            r = 0.5 / max(dims)  # 8,000 particles: r = 0.025, the block fills the cube
            p.update(boundary=0, radius=r, has_cube=1, cube_min=(0.0, 0.0, 0.0), cube_max=(1.0, 1.0, 1.0))
            return [(_block(r, (0.0, 0.0, 0.0), dims), None, p)]
        r = 0.25 / max(dims)
        p.update(boundary=2, radius=r, bvisc=0.01)
        return [(_block(r, (2 * r, 2 * r, 2 * r), dims), sph_gb300.sample_box(4 * r, (0.0, 0.0, 0.0), (1.0, 0.8, 0.8)), p)]
    if kind == "dam":
        dims = _ragged(case["n"])
        r = 0.25 / dims[0]
        b = [sph_gb300.sample_box(4 * r, (0.0, 0.0, 0.0), (1.5, 0.8, 0.8))]
        p = dict(workloads.DFSPH, radius=r)
        if case["forces"]:
            b.append(sph_gb300.sample_sphere(r, (1.0, 0.3, 0.4), 0.12))
            p.update(visc_method=2, visc=0.01, bvisc=0.01, st_method=3, st=0.5, adh_method=4, adh=0.1)
        return [(_block(r, (2 * r, 2 * r, 2 * r), dims), np.concatenate(b), p)]
    if kind == "drop":
        x, b, p, _ = workloads.pcisph_drop(case["radius"])
        return [(x, b, p)]
    return [(x, b, p) for x, b, p, _ in workloads.batched_mix(case["scenes"])]


def _disturbed(case, seed):
    """_geometry with the seed's jitter and velocities: [(x, v, boundary, parameters)]."""
    rng = np.random.default_rng([seed, 20])
    out = []
    for x, b, p in _geometry(case):
        r = p["radius"]
        if case["kind"] == "drop":
            # the pool at rest, the drop falling (at 0.6 m it reaches the pool with 3.4 m/s)
            x = x + rng.uniform(-0.01 * r, 0.01 * r, x.shape)
            v = np.zeros_like(x)
            v[x[:, 1] > 0.3, 1] = -rng.uniform(1.0, 3.0)
        else:
            x = x + rng.uniform(-0.02 * r, 0.02 * r, x.shape)
            c = x.mean(axis=0)
            v = rng.uniform(-0.5, 0.5, 3) + np.cross(rng.uniform(-1.0, 1.0, 3), x - c)
            v[:, 1] -= rng.uniform(0.0, 0.5)
        out.append((np.ascontiguousarray(x), np.ascontiguousarray(v), b, dict(p, precision=case["precision"])))
    return out


# ---- the measured calls --------------------------------------------------------------------------------------------

def prepare(case, seed):
    scenes = _disturbed(case, seed)
    if case["kind"] != "mix":
        x, v, b, p = scenes[0]
        s = sph_gb300.Scene(**p)
        s.set_fluid(x, v)
        if b is not None:
            s.add_boundary_points(b)
        s.init()
        s.set_graph(case["graph"])
        return dict(case=case, scene=s)
    n, nb = sum(t[0].shape[0] for t in scenes), sum(t[2].shape[0] for t in scenes)
    pool = sph_gb300.Pool(max_particles=n, max_boundary=nb, max_keys=65536 * len(scenes), max_scenes=len(scenes) + 1)
    # the launch shapes the autotuner picks for the mix on this card, so that no step is spent on measuring shapes
    pool.set_autotune(0)
    pool.set_tuning(build_block=256, build_occupancy=1024, queue_depth=40, solver_block=128, solver_occupancy=2048,
                    scan_width=16)
    pool.set_graph(case["graph"])
    ids = [pool.add_scene(x, v=v, boundary_points=b, steps=2**31 - 1, **p) for x, v, b, p in scenes]
    # pinned result buffers of every scene's positions and velocities, kept by the program
    out = [torch.empty((n, 3), dtype=torch.float64, pin_memory=torch.cuda.is_available()) for _ in range(2)]
    views, at = [], 0
    for t in scenes:
        views.append([o.numpy()[at:at + t[0].shape[0]] for o in out])
        at += t[0].shape[0]
    return dict(case=case, pool=pool, ids=ids, out=out, views=views)


def run(state):
    case = state["case"]
    if case["kind"] == "mix":
        pool = state["pool"]
        pool.step(case["steps"])
        for sid, (x, v) in zip(state["ids"], state["views"]):
            pool.get(sid, "x", out=x)
            pool.get(sid, "v", out=v)
        x, v = state["out"]
        return {"x": x.to(torch.float32), "v": v.to(torch.float32)}
    s = state["scene"]
    s.step(case["steps"])
    kind = torch.float64 if case["precision"] == "f64" else torch.float32
    return {f: torch.from_numpy(s.get(f)).to(kind) for f in ("x", "v", "rho")}


PAIRS = 30.0  # neighbours of a particle inside the fluid, spacing 2r and support 4r
# flops per pair and step: kernel value and gradient 34, each sum over the neighbours 8 (DFSPH: density with alpha,
# then 8 sums at its usual 2 + 1 iterations; PCISPH: 3 iterations of a density and a Spiky force; forces 60)
PAIR_FLOPS = {"wcsph": 34 + 8 + 34 + 20, "dam": 34 + 8 * 8, "mix": 34 + 8 * 8, "drop": 34 + 60 + 3 * 60}


def work(case):
    n = nb = 0
    for x, b, _ in _geometry(case):
        n += x.shape[0]
        nb += 0 if b is None else b.shape[0]
    size = 8 if case["precision"] == "f64" else 4
    # each step reads positions and velocities and writes them and the densities, and reads the boundary points and
    # weights once; the state is handed out once in float64
    step_bytes = (n * (6 + 7) + nb * 4) * size
    fields = 6 if case["kind"] == "mix" else 7
    flops = PAIR_FLOPS[case["kind"]] + (60 if case.get("forces") else 0)
    return {"bytes": case["steps"] * step_bytes + n * fields * 8, "flops": case["steps"] * n * PAIRS * flops}


# ---- the same steps in 64 bits with plain torch ----------------------------------------------------------------------
#
# Every sum over neighbours is a sum over the second axis of an (n, k) table of neighbour indices; the scenes of a mix
# are advanced together with a scene index per particle and the solver's scalars held per scene.

class _Near:
    """The points of y within `reach` of each x among the 27 cells (edge h) around it: idx (n, k), ok (n, k)."""

    def __init__(self, x, sx, y, sy, h, reach):
        cx, cy = torch.floor(x / h).long(), torch.floor(y / h).long()
        lo = torch.minimum(cx.amin(0), cy.amin(0)) - 2
        dim = torch.maximum(cx.amax(0), cy.amax(0)) + 3 - lo

        def key(c, s):
            c = c - lo
            return ((s * dim[0] + c[:, 0]) * dim[1] + c[:, 1]) * dim[2] + c[:, 2]

        ky, order = torch.sort(key(cy, sy), stable=True)
        ii, jj = [], []
        every = torch.arange(x.shape[0], device=x.device)
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                k = key(cx + torch.tensor([dx, dy, 0], device=x.device), sx)
                a, e = torch.searchsorted(ky, k - 1), torch.searchsorted(ky, k + 1, right=True)
                cnt = e - a
                i = torch.repeat_interleave(every, cnt)
                at = torch.arange(i.shape[0], device=x.device) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
                j = order[a[i] + at]
                near = ((x[i] - y[j]) ** 2).sum(1) <= reach * reach * (1 + 1e-12)
                ii.append(i[near])
                jj.append(j[near])
        i, j = torch.cat(ii), torch.cat(jj)
        i, by = torch.sort(i, stable=True)
        cnt = torch.bincount(i, minlength=x.shape[0])
        at = torch.arange(i.shape[0], device=x.device) - (torch.cumsum(cnt, 0) - cnt)[i]
        width = max(1, int(cnt.max()) if cnt.numel() else 1)
        self.idx = torch.zeros((x.shape[0], width), dtype=torch.long, device=x.device)
        self.ok = torch.zeros((x.shape[0], width), dtype=torch.bool, device=x.device)
        self.idx[i, at] = j[by]
        self.ok[i, at] = True


def _cubic(near, x, y, h):
    """(W, grad W) of the cubic spline for the table's pairs; zero outside it."""
    r = x[:, None] - y[near.idx]
    d = r.square().sum(2).sqrt()
    q = d / h
    k, l = 8 / (math.pi * h**3), 48 / (math.pi * h**3)
    in1, half = near.ok & (q <= 1), q <= 0.5
    w = torch.where(in1, torch.where(half, k * (6 * q**3 - 6 * q**2 + 1), k * 2 * (1 - q) ** 3), 0.0)
    g = torch.where(half, l * q * (3 * q - 2), -l * (1 - q) ** 2) / (d * h)
    g = torch.where(in1 & (d > 1e-5), g, 0.0)
    return w, g[..., None] * r, r, d, in1


class _Exact:
    def __init__(self, case, seed):
        self.case = case
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        scenes = _disturbed(case, seed)
        as_t = lambda parts: torch.from_numpy(np.concatenate(parts)).to(dev)  # noqa: E731
        self.x, self.v = as_t([t[0] for t in scenes]), as_t([t[1] for t in scenes])
        self.sid = as_t([np.full(t[0].shape[0], k) for k, t in enumerate(scenes)])
        self.S, self.n = len(scenes), self.x.shape[0]
        self.per = torch.bincount(self.sid, minlength=self.S).double()
        p = self.p = scenes[0][3]  # one parameter set per case
        self.h, self.rho0 = 4 * p["radius"], 1000.0
        self.m = self.rho0 * (2 * p["radius"]) ** 3
        self.g = torch.tensor([0.0, -9.81, 0.0], dtype=torch.float64, device=dev)
        self.b = None
        if p["boundary"] == 2:
            self.b = as_t([t[2] for t in scenes])
            self.bsid = as_t([np.full(t[2].shape[0], k) for k, t in enumerate(scenes)])
            near = _Near(self.b, self.bsid, self.b, self.bsid, self.h, self.h)
            self.bw = self.rho0 / _cubic(near, self.b, self.b, self.h)[0].sum(1)
        self.a = torch.zeros_like(self.x)
        self.dt = torch.full((self.S,), p.get("dt", 1e-4), dtype=torch.float64, device=dev)
        self.its = torch.zeros(self.S, dtype=torch.long, device=dev)
        self.kappa = torch.zeros(self.n, dtype=torch.float64, device=dev)
        self.max_error = 0.0

    def find(self, reach=1.0):
        self.near = _Near(self.x, self.sid, self.x, self.sid, self.h, reach * self.h)
        if self.b is not None:
            self.bnear = _Near(self.x, self.sid, self.b, self.bsid, self.h, reach * self.h)

    def density_terms(self):
        """Densities, m grad W per pair, and the boundary's summed weighted gradient."""
        w, g, _, _, _ = _cubic(self.near, self.x, self.x, self.h)
        self.rho = self.m * w.sum(1)
        self.G = self.m * g
        self.bg = torch.zeros_like(self.x)
        if self.b is not None:
            w, g, _, _, _ = _cubic(self.bnear, self.x, self.b, self.h)
            bw = self.bw[self.bnear.idx]
            self.rho = self.rho + (bw * w).sum(1)
            self.bg = (bw[..., None] * g).sum(1)

    def forces(self):
        """Viscosity, surface tension and adhesion added to the accelerations."""
        p, h, m, rho, i = self.p, self.h, self.m, self.rho, self.near.idx
        w, g, r, d, ok = _cubic(self.near, self.x, self.x, h)
        dt, rhoj, dv = self.dt[self.sid][:, None], rho[i], self.v[i] - self.v[:, None]
        visc, bvisc = p.get("visc", 0.0), p.get("bvisc", 0.0)
        lapl = 45 / (math.pi * h**6)
        if p.get("visc_method", -1) == 2:
            self.a += ((visc * m / rhoj * w)[..., None] * dv).sum(1) / dt
        elif p.get("visc_method", -1) == 0:
            self.a += visc / self.rho0 * ((torch.where(ok, lapl * (h - d), 0.0) * m / rhoj)[..., None] * dv).sum(1)
        if self.b is not None:
            bw_, bg_, br, bd, bok = _cubic(self.bnear, self.x, self.b, h)
            bw = self.bw[self.bnear.idx]
            if bvisc and p["visc_method"] == 2:
                self.a -= self.v * (bvisc * bw / rho[:, None] * bw_).sum(1)[:, None] / dt
        if p.get("st", 0.0):
            nrm = h * ((m / rhoj)[..., None] * g).sum(1)
            c1, c2 = 32 / (math.pi * h**9), h**6 / 64
            t = (h - d) ** 3 * d**3
            coh = torch.where(2 * d > h, c1 * t, torch.where(d > 0, 2 * c1 * t - c2, 0.0))
            on = ok & (d > 0)
            kij = p["st"] * 2 * self.rho0 / (rho[:, None] + rhoj)
            f = (-m * coh / torch.where(on, d, 1.0))[..., None] * r - (nrm[:, None] - nrm[i])
            self.a += (torch.where(on, kij, 0.0)[..., None] * f).sum(1)
        if p.get("adh", 0.0) and self.b is not None:
            val = torch.where(bok & (2 * bd > h), -4 * bd * bd / h + 6 * bd - 2 * h, 0.0).clamp_min(0).sqrt().sqrt()
            self.a -= ((p["adh"] * bw * val / torch.where(bok & (bd > 0), bd, 1.0))[..., None] * br).sum(1)

    # -- WCSPH
    def wcsph(self):
        self.find()
        self.density_terms()
        pr = (1000.0 * 1000.0 / 7.0 * ((self.rho / self.rho0) ** 7 - 1)).clamp_min(0)
        dp = pr / self.rho**2
        self.a -= ((dp[:, None] + dp[self.near.idx])[..., None] * self.G).sum(1) + dp[:, None] * self.bg
        self.forces()
        self.integrate(self.a + self.g)

    def integrate(self, acc):
        dt = self.p["dt"]
        self.v = self.v + acc * dt
        self.x = self.x + self.v * dt
        self.a = torch.zeros_like(self.a)
        if self.p.get("has_cube"):
            lo, hi = self.x < 0.0, self.x > 1.0
            self.v = torch.where((lo & (self.v < 0)) | (hi & (self.v > 0)), 0.0, self.v)
            self.x = self.x.clamp(0.0, 1.0)

    # -- PCISPH
    def pcisph(self):
        p, h, m, dt = self.p, self.h, self.m, self.p["dt"]
        self.find(1.2)
        self.density_terms()
        self.forces()
        grid = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64) * 2 * p["radius"]
        r = torch.cartesian_prod(grid, grid, grid)
        g = -945 / (32 * math.pi * h**9) * (h * h - (r * r).sum(1)).clamp_min(0)[:, None] ** 2 * r
        delta = 1 / (2 * (m * dt / self.rho0) ** 2 * float((g.sum(0) ** 2).sum() + (g * g).sum()))

        def spiky(near, y):
            r = self.x[:, None] - y[near.idx]
            d = r.square().sum(2).sqrt()
            on = near.ok & (d > 0) & (d <= h)
            return torch.where(on, -45 / (math.pi * h**6) * (h - d) ** 2 / torch.where(on, d, 1.0), 0.0)[..., None] * r

        sg, sb = spiky(self.near, self.x), (self.bw[self.bnear.idx][..., None] * spiky(self.bnear, self.b)).sum(1)
        press, pacc = torch.zeros_like(self.rho), torch.zeros_like(self.x)
        it, on = 0, self.max_error > p["eta"] or p["min_it"] > 0
        while on:
            pred = self.x + (self.v + (self.a + pacc + self.g) * dt) * dt
            rho = m * _cubic(self.near, pred, pred, h)[0].sum(1)
            rho = rho + (self.bw[self.bnear.idx] * _cubic(self.bnear, pred, self.b, h)[0]).sum(1)
            err = (rho - self.rho0).clamp_min(0)
            press = press + delta * err
            dp = press / rho**2
            pacc = -(m * (dp[:, None] + dp[self.near.idx])[..., None] * sg).sum(1) - dp[:, None] * sb
            self.rho, self.max_error, it = rho, float(err.max()) / self.rho0, it + 1
            on = (self.max_error > p["eta"] or it < p["min_it"]) and it < p["max_it"]
        self.integrate(self.a + self.g + pacc)

    # -- DFSPH
    def grid(self):
        self.find()
        self.density_terms()
        s = self.G.sum(1) + self.bg
        den = s.square().sum(1) + self.G.square().sum((1, 2))
        self.alpha = torch.where(den.abs() > 1e-5, self.rho / den, 0.0)

    def div(self):
        """sum_j m (v_i - v_j) . grad W_ij with the boundary's part."""
        return ((self.v[:, None] - self.v[self.near.idx]) * self.G).sum((1, 2)) + (self.v * self.bg).sum(1)

    def correct(self, k, on, boundary=1.0):
        ks = k[:, None] + k[self.near.idx]
        ks = torch.where(ks.abs() > 1e-5, ks, 0.0)
        kb = boundary * k
        kb = torch.where(kb.abs() > 1e-5, kb, 0.0)
        dv = self.dtp[:, None] * ((ks[..., None] * self.G).sum(1) + kb[:, None] * self.bg)
        self.v = self.v - torch.where(on[self.sid][:, None], dv, 0.0)

    def mean(self, e):
        return torch.zeros_like(self.per).index_add_(0, self.sid, e) / self.per / self.rho0

    def solve(self, error, limit, min_it, max_it, on_correct):
        on = torch.full((self.S,), min_it > 0 and max_it > 0, device=self.x.device)
        its = torch.zeros_like(self.its)
        e, k = error()
        while bool(on.any()):
            self.correct(k, on)
            on_correct(e, on[self.sid])
            e2, k2 = error()
            act = on[self.sid]
            e, k = torch.where(act, e2, e), torch.where(act, k2, k)
            its = its + on
            on = on & ((self.mean(e) > limit) | (its < min_it)) & (its < max_it)
        return its

    def dfsph(self):
        p, every = self.p, torch.ones(self.S, dtype=torch.bool, device=self.x.device)
        if p.get("visc") or p.get("st"):
            self.forces()
        dtp = self.dt[self.sid]
        speed = (self.v + (self.a + self.g) * dtp[:, None]).norm(dim=1).sqrt()
        vmax = torch.full_like(self.dt, 0.1).scatter_reduce_(0, self.sid, speed, "amax")
        cfl = p["cfl"] * 0.4 * 2 * p["radius"] / vmax
        self.dt = torch.where(cfl < self.dt, cfl, torch.where(self.its > 3, self.dt * 0.99, self.dt * 1.001))
        self.dt = self.dt.clamp(p["min_dt"], p["max_dt"])
        dt = self.dtp = self.dt[self.sid]
        self.v = self.v + (self.a + self.g) * dt[:, None]
        self.a = torch.zeros_like(self.a)
        self.correct((self.kappa / self.rho).clamp_max(1e-9) / dt**2, every, 2.0)
        self.kappa = torch.zeros_like(self.kappa)

        def density_error():
            e = (self.rho + self.div() * dt).clamp_min(self.rho0) - self.rho0
            return e, e * self.alpha / (dt * dt * self.rho)

        def add_kappa(e, act):
            self.kappa = self.kappa + torch.where(act, e * self.alpha, 0.0)

        self.its = self.solve(density_error, p["eta"], 2, p["max_it"], add_kappa)
        self.x = self.x + self.v * dt[:, None]
        self.grid()
        few = (self.G.square().sum(2) > 0).sum(1) < 20

        def div_error():
            e = torch.where(few, 0.0, self.div().clamp_min(0))
            return e, e * self.alpha / (dt * self.rho)

        self.solve(div_error, p["eta_v"] / self.dt, 1, p["max_it"], lambda e, act: None)

    def run(self):
        step = {DFSPH: self.dfsph, WCSPH: self.wcsph, PCISPH: self.pcisph}[self.p["method"]]
        if self.p["method"] == DFSPH:
            self.grid()
        for _ in range(self.case["steps"]):
            step()
        out = {"x": self.x, "v": self.v, "rho": self.rho}
        if self.case["kind"] == "mix":
            del out["rho"]
        return out


def exact(case, seed):
    return _Exact(case, seed).run()
