"""
What is timed: calls that a user of this package makes, through its public entry points, over
the range of sizes, types and options that the path is used with.

A case is a dict of plain values. Its "kind" says which entry points it goes through:

  run     Simulation.run: many steps in one call, the way a simulation is advanced
  loop    update_E, a soft source, update_H, update_S: the driver loop of the reference
  batch   BatchSimulation.run: a sweep of cavity variants of uneven sizes
  layer   Simulation.run with a learned boundary layer attached (its inference every step)
  train   one optimisation step of a boundary network (forward, backward, Adam)
"""
from __future__ import annotations

import math

import numpy
import torch

from opencl_fdtd_gb300 import Simulation
from opencl_fdtd_gb300 import learned_boundary
from opencl_fdtd_gb300.batch import BatchSimulation

DT = 0.99 / math.sqrt(3)
LEARN_RATE = 2e-3


def _run(name, shape, steps, **kw):
    case = {"name": name, "kind": "run", "nx": shape[0], "ny": shape[1], "nz": shape[2], "steps": steps,
            "dtype": "f32", "poynting": True, "faces": "all", "thickness": 8, "grid": "unit", "mu": False,
            "bloch": False, "monitor": False}
    case.update(kw)
    return case


def listed():
    return [
        # a unit-cell sized trial grid, as the parity fixtures use: only launches and latency
        _run("run_24", (24, 24, 24), 20, poynting=False, thickness=4),
        # the 64^3 slab workload (fields fit the L2), a stretch of its 500 steps
        _run("run_64", (64, 64, 64), 50, poynting=False),
        # the benchmark grid: a photonic-crystal cavity with its point monitor, ten steps a call
        _run("run_cavity", (395, 345, 73), 10, monitor=True),
        # the same grid through the per-call loop that a program of the reference runs
        {"name": "loop_cavity", "kind": "loop", "nx": 395, "ny": 345, "nz": 73, "steps": 2, "dtype": "f32",
         "poynting": True, "faces": "all", "thickness": 8, "grid": "unit", "mu": False, "bloch": False,
         "monitor": False},
        # an odd grid with graded cells, magnetic materials, absorbers on three faces only, and an
        # odd number of steps
        _run("run_graded", (151, 129, 61), 11, faces="mixed", thickness=6, grid="table", mu=True),
        # double precision, for convergence studies
        _run("run_f64", (197, 173, 73), 8, dtype="f64"),
        # a periodic cell at a Bloch wave vector: split complex fields, eps and mu, absorbers on z
        _run("run_bloch", (128, 128, 256), 5, poynting=False, faces="z", mu=True, bloch=True),
        # a cube, with z rows much longer than those of a slab
        _run("run_cube", (300, 300, 300), 4),
        # a sweep of cavity variants stepped together, float32 and 16-bit storage
        {"name": "batch_f32", "kind": "batch", "variants": 8, "storage": "f32", "lo": 96, "hi": 224, "steps": 10},
        {"name": "batch_bf16u", "kind": "batch", "variants": 8, "storage": "bf16u", "lo": 96, "hi": 224, "steps": 10},
        # a cavity whose absorbers are replaced by the two-cell learned layer on all faces
        {"name": "layer_bf16x2", "kind": "layer", "nx": 203, "ny": 177, "nz": 61, "steps": 5,
         "precision": "bf16x2", "poynting": True},
        # one optimisation step at the batch size that the training loop uses
        {"name": "train_4096", "kind": "train", "batch": 4096},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _shape(rng, cells):
    """Three extents, z the shortest more often than not, of about that many cells."""
    nz = int(min(max(round(_log(rng, 12, 320)), 12), max(12, cells // 400)))
    skew = rng.uniform(0.7, 1.4)
    nx = max(12, int(round(math.sqrt(cells / nz) * skew)))
    ny = max(12, int(round(cells / nz / nx)))
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "run", "loop", "batch", "layer", "train"])
    if kind in ("run", "loop"):
        bloch = kind == "run" and rng.random() < 0.2
        f64 = rng.random() < 0.15
        cells = _log(rng, 1e4, 4e6 if bloch or f64 else 1.2e7)
        nx, ny, nz = _shape(rng, cells)
        steps = max(1, min(rng.randint(1, 40), int(3e7 / (nx * ny * nz))))
        if kind == "loop":
            steps = min(steps, 3)
        case = _run("", (nx, ny, nz), steps, dtype="f64" if f64 else "f32",
                    poynting=kind == "loop" or (not bloch and rng.random() < 0.7),
                    faces="z" if bloch else rng.choice(["all", "all", "z", "mixed", "none"]),
                    thickness=min(rng.choice([4, 6, 8, 8, 10]), min(nx, ny, nz) // 3),
                    grid=rng.choice(["unit", "unit", "half", "table"]), mu=rng.random() < 0.25, bloch=bloch,
                    monitor=kind == "run" and rng.random() < 0.3)
        case["kind"] = kind
        del case["name"]
        return case
    if kind == "batch":
        lo = rng.randint(48, 110)
        return {"kind": "batch", "variants": rng.randint(2, 8), "storage": rng.choice(["f32", "f32", "bf16u", "fp16"]),
                "lo": lo, "hi": rng.randint(lo + 8, 220), "steps": rng.randint(2, 10)}
    if kind == "layer":
        return {"kind": "layer", "nx": rng.randint(40, 260), "ny": rng.randint(40, 220), "nz": rng.randint(24, 120),
                "steps": rng.randint(1, 5), "precision": rng.choice(["bf16x2", "bf16x2", "linear", "bf16"]),
                "poynting": rng.random() < 0.7}
    return {"kind": "train", "batch": int(_log(rng, 200, 16384))}


# ---- inputs -----------------------------------------------------------------------------------
def _dtype(case):
    return numpy.float64 if case["dtype"] == "f64" else numpy.float32


def _slab(shape, rng, dtype):
    """A dielectric slab in the middle of z with a jittered lattice of air holes, and a small
    metal block."""
    nx, ny, nz = shape
    a, r = rng.uniform(8, 12), rng.uniform(2.2, 3.4)
    x = (numpy.arange(nx) + rng.uniform(0, a)) % a - a / 2
    y = (numpy.arange(ny) + rng.uniform(0, a)) % a - a / 2
    holes = x[:, None] ** 2 + y[None, :] ** 2 < r * r
    t = max(1, nz // 24)
    sl = slice(nz // 2 - t, nz // 2 + t)
    eps = []
    for _ in range(3):
        e = numpy.ones(shape, dtype)
        e[:, :, sl] = numpy.where(holes, 1.0, 12.11)[:, :, None]
        e[nx // 3:nx // 3 + 2, ny // 3:ny // 3 + 2, nz // 3:nz // 3 + 2] = numpy.inf
        eps.append(e)
    return eps


def _mu(shape, rng, dtype):
    out = []
    for _ in range(3):
        m = numpy.ones(shape, dtype)
        m[shape[0] // 4:shape[0] // 2, :, shape[2] // 4:shape[2] // 2] = rng.uniform(1.1, 2.0)
        out.append(m)
    return out


def _faces(case):
    T = case["thickness"]
    names = {"all": ["xn", "xp", "yn", "yp", "zn", "zp"], "z": ["zn", "zp"], "mixed": ["xn", "yp", "zp"],
             "none": []}[case["faces"]]
    return [{"axis": n[0], "polarity": n[1], "thickness": T} for n in names] if T else []


def _wave(steps):
    return [math.sin(0.3 * t + 0.2) * math.exp(-0.5 * ((t - 12) / 8) ** 2) for t in range(steps)]


def _fill(fields, seed):
    """Small random values in fields that live on the GPU, by the seed alone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7 + 1)
    for f in fields:
        f.copy_(torch.randn(f.shape, generator=gen, device="cuda", dtype=torch.float32) * 1e-2)


def _grid_inputs(case, seed):
    shape = (case["nx"], case["ny"], case["nz"])
    rng = numpy.random.default_rng(seed)
    dtype = _dtype(case)
    kw = dict(epsilon=_slab(shape, rng, dtype), pmls=_faces(case), do_poynting=case["poynting"], float_type=dtype)
    if case["mu"]:
        kw["mu"] = _mu(shape, rng, dtype)
    if case["grid"] == "half":
        kw["dxes"] = 0.5
    elif case["grid"] == "table":
        kw["dxes"] = [[rng.uniform(0.8, 1.25, n) for n in shape] for _ in range(2)]
    if case["bloch"]:
        kw["bloch_boundaries"] = [{"axis": "x", "real": math.cos(0.3 * math.pi), "imag": math.sin(0.3 * math.pi)},
                                  {"axis": "y", "real": math.cos(0.1 * math.pi), "imag": math.sin(0.1 * math.pi)}]
    centre = tuple(s // 2 for s in shape)
    N = shape[0] * shape[1] * shape[2]
    return shape, kw, int(numpy.ravel_multi_index(centre, shape)) + N


def _monitor_points(shape):
    c = [s // 2 for s in shape]
    d = min(20, min(c) - 1)
    return [(1, c), (1, [c[0] + d, c[1], c[2]]), (1, [c[0] - d, c[1], c[2]]), (1, [c[0], c[1] + d, c[2]]),
            (1, [c[0], c[1] - d, c[2]])]


OMEGAS = (0.15, 0.1621, 0.175)


def _batch_shapes(case):
    """The variants' shapes: uneven, the same ones for every seed."""
    lo, hi = case["lo"], case["hi"]
    rng = numpy.random.default_rng(1000 * lo + hi)
    return [(int(rng.integers(lo, hi)), int(rng.integers(lo, hi)), int(rng.integers(lo // 2, lo // 2 + 26)))
            for _ in range(case["variants"])]


def _batch_case(shape):
    return _run("", shape, 0, poynting=False)


def _train_inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 13 + 5)
    B = case["batch"]
    X = torch.randn((B, learned_boundary.IN), generator=gen, device="cuda")
    X = X / X.square().mean(dim=1, keepdim=True).sqrt()
    A = torch.randn((learned_boundary.IN, learned_boundary.OUT), generator=gen, device="cuda") * 0.1
    return X.contiguous(), (X @ A).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "loop"):
        shape, kw, ind = _grid_inputs(case, seed)
        sim = Simulation(**kw)
        _fill([f for f in (sim.E, sim.H, sim.F, sim.G) if f is not None], seed)
        mon = sim.dft_monitor(_monitor_points(shape), OMEGAS, record=False) if case["monitor"] else None
        return {"kind": kind, "sim": sim, "ind": ind, "wave": _wave(case["steps"]), "monitor": mon,
                "steps": case["steps"]}
    if kind == "batch":
        sims, src = [], []
        for v, shape in enumerate(_batch_shapes(case)):
            _, kw, ind = _grid_inputs(_batch_case(shape), seed + v)
            sim = Simulation(**kw)
            _fill([sim.E, sim.H], seed + 31 * v)
            sims.append(sim)
            src.append([(ind, _wave(200))])
        batch = BatchSimulation(sims, storage=case["storage"], sources=src, steps=200)
        return {"kind": kind, "batch": batch, "sims": sims, "steps": case["steps"]}
    if kind == "layer":
        shape, kw, ind = _grid_inputs(_run("", (case["nx"], case["ny"], case["nz"]), 0, faces="none",
                                           poynting=case["poynting"]), seed)
        net = learned_boundary.BoundaryNet(seed=seed, memory=(1.0 - DT) / (1.0 + DT))
        for f in range(6):
            net.embed_linear(f, learned_boundary.mur_map(f))
        sim = Simulation(dt=net.dt, **kw)
        _fill([sim.E, sim.H], seed)
        layer = learned_boundary.LearnedBoundary(net, case["precision"])
        layer.attach(sim)
        return {"kind": kind, "sim": sim, "ind": ind, "wave": _wave(case["steps"]), "monitor": None,
                "steps": case["steps"], "layer": layer}
    X, T = _train_inputs(case, seed)
    return {"kind": "train", "net": learned_boundary.BoundaryNet(seed=seed), "X": X, "T": T, "face": seed % 6}


# ---- one pass -----------------------------------------------------------------------------------
def _fields(sim, names="EHFGS"):
    return {k: getattr(sim, k) for k in names if getattr(sim, k) is not None}


def run(state):
    kind = state["kind"]
    if kind in ("run", "layer"):
        sim, mon = state["sim"], state["monitor"]
        sim.run(state["steps"], point_sources=[(state["ind"], state["wave"])], monitor=mon)
        out = _fields(sim)
        if mon is not None:
            out["spectrum"] = mon.accum
        return out
    if kind == "loop":
        sim, ind = state["sim"], state["ind"]
        for v in state["wave"]:
            sim.update_E([])
            sim.E[ind] += v
            e = sim.update_H([])
            sim.update_S([e])
        return _fields(sim)
    if kind == "batch":
        state["batch"].run(state["steps"])
        state["batch"].sync()
        return [_fields(s, "EH") for s in state["sims"]]
    net, face = state["net"], state["face"]
    loss, grad = net.gradient(face, state["X"], state["T"])
    net.adam_step(face, grad, LEARN_RATE)
    return {"loss": loss, "grad": grad, "params": net.params[face], "m": net.m[face], "v": net.v[face]}


# ---- what a pass cannot do without ----------------------------------------------------------------
def _face_cells(case):
    n = {"x": case["nx"], "y": case["ny"], "z": case["nz"]}
    cells = case["nx"] * case["ny"] * case["nz"]
    return sum(f["thickness"] * cells // n[f["axis"]] for f in _faces(case))


def _grid_work(case, steps, elem):
    """A step reads E, H and dt/eps (and dt/mu), writes E, H (and S), and reads and writes the four
    auxiliary values of each absorbing cell of a face; a Bloch pair has twice the fields."""
    cells = case["nx"] * case["ny"] * case["nz"]
    pair = 2 if case["bloch"] else 1
    values = 12 * pair + 3 + (3 if case["mu"] else 0) + (3 if case["poynting"] else 0)
    spacing = 12 * pair if case["grid"] != "unit" else 0
    flops = 36 * pair + spacing + (27 if case["poynting"] else 0)
    fc = _face_cells(case)
    return {"bytes": float(steps * elem * (values * cells + 8 * pair * fc)),
            "flops": float(steps * (flops * cells + 20 * pair * fc))}


def work(case):
    kind = case["kind"]
    if kind in ("run", "loop"):
        return _grid_work(case, case["steps"], 8 if case["dtype"] == "f64" else 4)
    if kind == "batch":
        out = {"bytes": 0.0, "flops": 0.0}
        for shape in _batch_shapes(case):
            c = _batch_case(shape)
            w = _grid_work(c, case["steps"], 4 if case["storage"] == "f32" else 2)
            out["flops"] += w["flops"]
            # the auxiliary arrays stay in float32; 16-bit storage is read back once a pass
            out["bytes"] += w["bytes"] + (0 if case["storage"] == "f32" else
                                          16 * case["steps"] * _face_cells(c) + 36 * shape[0] * shape[1] * shape[2])
        return out
    if kind == "layer":
        w = _grid_work(_run("", (case["nx"], case["ny"], case["nz"]), 0, faces="none", poynting=case["poynting"]),
                       case["steps"], 4)
        columns = 2 * (case["nx"] * case["ny"] + case["nx"] * case["nz"] + case["ny"] * case["nz"])
        per = 2 * 108 * 6 if case["precision"] == "linear" else 2 * (108 * 64 + 64 * 64 + 64 * 6)
        return {"bytes": w["bytes"] + case["steps"] * columns * 2 * 24.0, "flops": w["flops"] + float(case["steps"] * columns * per)}
    B, P = case["batch"], 108 * 64 + 64 * 64 + 64 * 6
    return {"bytes": 4.0 * (B * (108 + 6) + 11526 * 7), "flops": 2.0 * B * (3 * P - 108 * 64) + 12.0 * 11526}


# ---- the same in 64 bits ---------------------------------------------------------------------------
def _tables(face, dt):
    """CPML coefficients of a face by depth from the outside, for the E and the H update."""
    T, m = face["thickness"], 3.5
    sigma_max = 1.6 / 2 * (m + 1)

    def coefficients(depth):
        sigma = (depth / T) ** m * sigma_max
        p0 = numpy.exp(-sigma * dt)
        return p0, p0 - 1.0

    deep = numpy.arange(T, 0, -1).astype(numpy.float64)
    half = deep - 0.5
    return (coefficients(half), coefficients(deep)) if face["polarity"] == "p" else (coefficients(deep), coefficients(half))


def _along(values, axis):
    shape = [1, 1, 1]
    shape[axis] = len(values)
    return torch.as_tensor(numpy.ascontiguousarray(values), dtype=torch.float64, device="cuda").view(shape)


class _Grid64:
    """The Yee step with CPML, graded cells, diagonal materials and Bloch phases on whole arrays."""

    def __init__(self, shape, kw, fields, dt=None):
        self.shape = shape
        dx = kw.get("dxes", 1.0)
        if isinstance(dx, float):
            self.spacing = [[_along([dx], a) for a in range(3)]] * 2
            smallest = dx
        else:
            rounded = [[(1.0 / (1 / numpy.asarray(v)).astype(kw["float_type"]).astype(numpy.float64)) for v in g] for g in dx]
            self.spacing = [[_along(v, a) for a, v in enumerate(g)] for g in rounded]
            smallest = min(float(v.min()) for g in dx for v in g)
        self.dt = smallest * 0.99 / math.sqrt(3) if dt is None else dt
        put = lambda a: torch.from_numpy(a).to("cuda").to(torch.float64)  # noqa: E731
        self.ce = [self.dt / put(e) for e in kw["epsilon"]]
        self.ch = [self.dt / put(m) for m in kw["mu"]] if "mu" in kw else [self.dt] * 3
        self.phase = [None] * 3
        for b in kw.get("bloch_boundaries", ()):
            self.phase["xyz".index(b["axis"])] = complex(b["real"], b["imag"])
        kind = torch.complex128 if any(p is not None for p in self.phase) else torch.float64
        split = {k: [c.to(torch.float64) for c in f.view(3, *shape)] for k, f in fields.items()}
        self.E, self.H = ([torch.complex(a, b) for a, b in zip(split[p], split[q])] if q in split else split[p]
                          for p, q in (("E", "F"), ("H", "G")))
        self.S = None
        self.faces = []
        for f in kw["pmls"]:
            a, T = "xyz".index(f["axis"]), f["thickness"]
            cut = [slice(None)] * 3
            cut[a] = slice(0, T) if f["polarity"] == "n" else slice(shape[a] - T, shape[a])
            flip = (lambda v: v) if f["polarity"] == "n" else (lambda v: v[::-1])
            tabs = [[_along(flip(v), a) for v in t] for t in _tables(f, self.dt)]
            psi = [[torch.zeros([T if r == a else shape[r] for r in range(3)], dtype=kind, device="cuda")
                    for _ in range(2)] for _ in range(2)]
            self.faces.append((a, tuple(cut), tabs, psi))

    def _shift(self, f, axis, up, phase=True):
        """The neighbour one cell up or down the axis, across the periodic edge."""
        n = torch.roll(f, -1 if up else 1, axis)
        if phase and self.phase[axis] is not None:
            edge = [slice(None)] * 3
            edge[axis] = -1 if up else 0
            n[tuple(edge)] *= self.phase[axis] if up else self.phase[axis].conjugate()
        return n

    def _curl(self, F, up):
        """Curl with forward (up) or backward differences, the absorbers' terms in it."""
        which, step = (1, self.spacing[0]) if up else (0, self.spacing[1])
        out = [torch.zeros_like(F[0]) for _ in range(3)]
        for r in range(3):
            u, v = [c for c in range(3) if c != r]
            for c, into in ((u, v), (v, u)):
                near = self._shift(F[c], r, up)
                d = ((near - F[c]) if up else (F[c] - near)) / step[r]
                for a, cut, tabs, psi in self.faces:
                    if a != r:
                        continue
                    p0, p1 = tabs[which]
                    q = psi[which][0 if c == u else 1]
                    q.mul_(p0).add_(p1 * d[cut])
                    d[cut] += q
                # curl_into has + d_r F_c for (into, r, c) an even permutation
                if (into, r, c) in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
                    out[into] += d
                else:
                    out[into] -= d
        return out

    def step(self, index, value, layer=None):
        ghosts = layer.predict(self) if layer else None
        for c, k in enumerate(self._curl(self.H, False)):
            self.E[c] = self.E[c] + self.ce[c] * k
        if layer:
            layer.fix(self, ghosts, 0)
        cells = self.shape[0] * self.shape[1] * self.shape[2]
        self.E[index // cells].view(-1)[index % cells] += value
        old = self.H
        self.H = [h - ch * k for h, ch, k in zip(self.H, self.ch, self._curl(self.E, True))]
        self.both = [a + b for a, b in zip(self.H, old)]
        if layer:
            layer.fix(self, ghosts, 1)

    def poynting(self):
        """The Poynting vector of the last step, averaged to the cells."""
        A = self.both
        sums = {(c, r): self._shift(self.E[c], r, True) + self.E[c] for c in range(3) for r in range(3) if c != r}
        out = []
        for r in range(3):
            u, v = (r + 1) % 3, (r + 2) % 3
            p = sums[u, r] * A[v]
            q = -sums[v, r] * A[u]
            out.append((p + q + self._shift(p, u, False) + self._shift(q, v, False)) * (self.dt / 8))
        return out


class _Layer64:
    """Mur's first-order condition as ghost fields outside the six faces."""

    def __init__(self):
        self.m = (1.0 - DT) / (1.0 + DT)
        self.ghosts = {}

    @staticmethod
    def _clamped(plane, axis, up):
        n = plane.shape[axis]
        index = torch.arange(n, device="cuda") + (1 if up else -1)
        return plane.index_select(axis, index.clamp(0, n - 1))

    def predict(self, g):
        for a in range(3):
            for side in range(2):
                F, other = (g.H, g.E) if side == 0 else (g.E, g.H)
                at = 0 if side == 0 else g.shape[a] - 1
                inner = 1 if side == 0 else g.shape[a] - 2
                for p in range(3):
                    if p == a:
                        continue
                    curl = 0.0
                    for r in range(3):
                        for q in range(3):
                            if len({p, r, q}) < 3:
                                continue
                            sign = 1.0 if (p, r, q) in ((0, 1, 2), (1, 2, 0), (2, 0, 1)) else -1.0
                            own = other[q].select(a, at)
                            if r == a:
                                near = other[q].select(a, inner)
                            else:
                                near = self._clamped(own, r - (1 if r > a else 0), side == 0)
                            curl = curl + sign * ((near - own) if side == 0 else (own - near))
                    ghost = (1.0 - self.m) * F[p].select(a, at) + (DT * curl if side == 0 else -self.m * DT * curl)
                    if (a, side, p) in self.ghosts:
                        ghost = ghost + self.m * self.ghosts[a, side, p]
                    self.ghosts[a, side, p] = ghost
        return self.ghosts

    def fix(self, g, ghosts, side):
        # every term from the fields as the update left them
        F, other, coef = (g.E, g.H, g.ce) if side == 0 else (g.H, g.E, [torch.full(g.shape, g.dt, dtype=torch.float64, device="cuda")] * 3)
        for a in range(3):
            at, across = (0, g.shape[a] - 1) if side == 0 else (g.shape[a] - 1, 0)
            for q in range(3):
                if q == a:
                    continue
                p = 3 - a - q
                sign = 1.0 if (q, a, p) in ((0, 1, 2), (1, 2, 0), (2, 0, 1)) else -1.0
                F[q].select(a, at).sub_(sign * coef[q].select(a, at) * (ghosts[a, side, p] - other[p].select(a, across)))


def _flat(parts):
    return torch.cat([p.reshape(-1) for p in parts])


def _exact_grid(case, seed, steps, layer=None, fill=None):
    shape, kw, ind = _grid_inputs(case, seed)
    n = 3 * shape[0] * shape[1] * shape[2]
    names = "EHFG" if case["bloch"] else "EH"
    fields = {k: torch.empty(n, dtype=torch.float64 if case["dtype"] == "f64" else torch.float32, device="cuda") for k in names}
    _fill(list(fields.values()), seed if fill is None else fill)
    g = _Grid64(shape, kw, fields, dt=DT if layer else None)
    mon, spectrum = _monitor_points(shape), None
    if case["monitor"]:
        spectrum = torch.zeros((len(mon), len(OMEGAS), 2), dtype=torch.float64)
    for t, v in enumerate(_wave(steps)):
        g.step(ind, float(kw["float_type"](v)), layer)
        if spectrum is not None:
            for i, (c, at) in enumerate(mon):
                x = complex(g.E[c][tuple(at)]).real
                for j, w in enumerate(OMEGAS):
                    ph = w * (t + 1) * g.dt
                    spectrum[i, j, 0] += x * math.cos(ph)
                    spectrum[i, j, 1] -= x * math.sin(ph)
    out = {}
    if case["bloch"]:
        out = {"E": _flat([c.real for c in g.E]), "F": _flat([c.imag for c in g.E]),
               "H": _flat([c.real for c in g.H]), "G": _flat([c.imag for c in g.H])}
    else:
        out = {"E": _flat(g.E), "H": _flat(g.H)}
    if case["poynting"]:
        out["S"] = _flat(g.poynting())
    if spectrum is not None:
        out["spectrum"] = spectrum
    return out


def _exact_train(case, seed):
    X, T = (v.double() for v in _train_inputs(case, seed))
    face, B = seed % 6, case["batch"]
    P = learned_boundary.BoundaryNet(seed=seed).params[face].double().requires_grad_(True)
    i, h, o = 108, 64, 6
    cut = numpy.cumsum([0, i * h, h, h * h, h, h * o, o])
    w1, b1, w2, b2, w3, b3 = (P[cut[k]:cut[k + 1]] for k in range(6))
    gelu = torch.nn.functional.gelu
    y = gelu(gelu(X @ w1.view(i, h) + b1) @ w2.view(h, h) + b2) @ w3.view(h, o) + b3
    axis, side = divmod(face, 2)
    wout = torch.zeros(6, dtype=torch.float64, device="cuda")
    for p in range(3):
        if p != axis:
            wout[p if side == 1 else 3 + p] = 1.0
    loss = ((y - T) ** 2 * wout).mean()
    grad, = torch.autograd.grad(loss, P)
    m, v = 0.1 * grad, 0.001 * grad * grad
    params = P.detach() - LEARN_RATE * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
    return {"loss": loss.detach(), "grad": grad, "params": params, "m": m, "v": v}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "loop"):
        return _exact_grid(case, seed, case["steps"])
    if kind == "batch":
        out = []
        for v, shape in enumerate(_batch_shapes(case)):
            out.append(_exact_grid(_batch_case(shape), seed + v, case["steps"], fill=seed + 31 * v))
        return out
    if kind == "layer":
        return _exact_grid(_run("", (case["nx"], case["ny"], case["nz"]), 0, faces="none", poynting=case["poynting"]),
                           seed, case["steps"], layer=_Layer64())
    return _exact_train(case, seed)
