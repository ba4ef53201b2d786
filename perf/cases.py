"""The work that programs have this library do, as measurable cases.

A pass of a step case is what a host program with an authoritative collection
does: the collection goes to the device from pinned host memory, the solver
advances it, and the fields the host reads come back to pinned host memory.
A pass of a search case sets new positions, searches, and reads the neighbor
lists into the program's own arrays; a pass of a render case renders one image
of the uploaded particles.
Every pass starts from the same uploaded collection, so passes repeat.

The scenes are this repository's breaking dams and search points
(fluidsolver_b200/scenes.py) in the units and settings of its benchmark
(spacing 1, rest density 1, IISPH time step 0.005, SESPH k 1000 and time step
0.001, viscosity 0.01). The dams are caught in mid-collapse: the column
flows outwards as it sinks, v = (a x, -a y, 0) with some noise, and the seed
draws the jitter of the positions and the noise.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from fluidsolver_b200 import (IISPHFluidSolver, IISPHFluidSolver3D, NeighborhoodSearch, ParticleCollection,
                              SESPHFluidSolver, SESPHFluidSolver3D, Timepoint, scenes)
from fluidsolver_b200 import _lib as F
from fluidsolver_b200.solver import BatchedIISPHFluidSolver3D

DT = {"sesph2d": 0.001, "iisph2d": 0.001, "sesph3d": 0.001, "iisph3d": scenes.REFERENCE_UNITS_DT,
      "batch": scenes.REFERENCE_UNITS_DT}
OUTPUTS = ("position", "velocity", "density", "pressure")


def listed():
    return [
        # The scale of the 2D scenarios: a hand-made dam, as a user of the 2D solvers starts with. Launches and
        # latency count. 20 steps between two looks at the result.
        dict(name="sesph2d_dam", kind="sesph2d", nx=50, ny=50, steps=20, search="hashed-2d", mode="fast"),
        # The same scale on the 2D IISPH solver with its default search, in the mode that repeats the reference's
        # arithmetic bit for bit (comparisons with the CPU solver).
        dict(name="iisph2d_dam_exact", kind="iisph2d", nx=50, ny=50, steps=10, search="quadratic-2d", mode="exact"),
        # A 2D scene ten times larger, of odd size: too many particles for the small-scene kernel.
        dict(name="sesph2d_40k", kind="sesph2d", nx=203, ny=197, steps=10, search="hashed-2d", mode="fast"),
        # One step of a small 3D scene through the solver interface's two calls, with the host collection
        # authoritative around it: what the Simulator does with entities and sensors on.
        dict(name="iisph3d_dropin_8k", kind="iisph3d", nx=20, ny=20, nz=20, steps=1, search="hashed-3d", mode="fast",
             calls="pair", layers=1),
        # The ordinary 3D dam.
        dict(name="iisph3d_dam_100k", kind="iisph3d", nx=40, ny=50, nz=50, steps=1, search="hashed-3d", mode="fast",
             calls="run", layers=1),
        # The headline dam: a million fluid particles and a quarter million boundary particles.
        dict(name="iisph3d_dam_1m", kind="iisph3d", nx=100, ny=100, nz=100, steps=1, search="hashed-3d", mode="fast",
             calls="run", layers=1),
        # The bit-exact mode at the ordinary size.
        dict(name="iisph3d_exact_100k", kind="iisph3d", nx=40, ny=50, nz=50, steps=2, search="hashed-3d", mode="exact",
             calls="run", layers=1),
        # The FP64 mode, the error reference for a scene of one's own; odd sizes, two boundary layers, the
        # compressed contract.
        dict(name="iisph3d_fp64_20k", kind="iisph3d", nx=31, ny=23, nz=29, steps=2, search="compressed-3d",
             mode="fp64", calls="run", layers=2),
        # The 3D SESPH solver at a size between the two dams.
        dict(name="sesph3d_250k", kind="sesph3d", nx=63, ny=63, nz=63, steps=1, search="hashed-3d", mode="fast",
             calls="run", layers=1),
        # A parameter sweep: many small dams of uneven size advanced together.
        dict(name="iisph3d_batch_64", kind="batch", count=64, smallest=2000, largest=60000, steps=1),
        # The neighborhood search on its own: points in, lists out (a program that wants the neighbor sets).
        dict(name="search_uniform_250k", kind="search", points="uniform", n=250_003, search="hashed-3d"),
        # A preview image of a dam.
        dict(name="render_dam_160x120", kind="render", nx=30, ny=40, nz=30, width=160, height=120, samples=1, depth=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape3(rng, lo, hi):
    f, a, b = _log(rng, lo, hi), rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
    nx, ny = max(6, round((f * a) ** (1 / 3))), max(6, round((f * b) ** (1 / 3)))
    return nx, ny, max(6, round(f / (nx * ny)))


def draw(rng):
    kind = rng.choice(["sesph2d", "iisph2d", "iisph3d", "iisph3d", "iisph3d", "sesph3d", "batch", "search", "render"])
    if kind in ("sesph2d", "iisph2d"):
        f, a = _log(rng, 900, 40000), rng.uniform(0.6, 1.6)
        nx = max(12, round(math.sqrt(f * a)))
        return dict(kind=kind, nx=nx, ny=max(12, round(f / nx)), steps=rng.randint(5, 20),
                    search=rng.choice(["hashed-2d", "quadratic-2d"]), mode=rng.choice(["fast", "fast", "exact"]))
    if kind in ("iisph3d", "sesph3d"):
        mode = rng.choice(["fast", "fast", "fast", "exact", "fp64"])
        nx, ny, nz = _shape3(rng, 2000, {"fast": 900_000, "exact": 150_000, "fp64": 60_000}[mode])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=1 if mode == "fast" else rng.randint(1, 4),
                    search=rng.choice(["hashed-3d", "hashed-3d", "quadratic-3d", "compressed-3d"]), mode=mode,
                    calls=rng.choice(["run", "pair"]), layers=rng.choice([1, 1, 2]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 64), smallest=2000, largest=_log(rng, 4000, 60000),
                    steps=1)
    if kind == "search":
        points = rng.choice(["uniform", "uniform", "blobs"])
        return dict(kind=kind, points=points, n=_log(rng, 5000, 250_000 if points == "uniform" else 120_000),
                    search=rng.choice(["hashed-3d", "quadratic-3d", "compressed-3d"]) if points == "uniform" else "hashed-3d")
    nx, ny, nz = _shape3(rng, 2000, 40000)
    return dict(kind="render", nx=nx, ny=ny, nz=nz, width=_log(rng, 40, 170), height=_log(rng, 40, 120),
                samples=rng.choice([1, 1, 2]), depth=rng.choice([2, 5, 10]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _flow(scene, seed, rate):
    """The dam's collection in mid-collapse (module docstring)."""
    col, nf = scene.collection, scene.n_fluid
    rng = np.random.default_rng(seed + 77)
    x = col.position[:nf]
    v = rng.normal(0.0, 0.02, x.shape).astype(np.float32)
    v[:, 0] += np.float32(rate) * x[:, 0]
    v[:, 1] -= np.float32(rate) * x[:, 1]
    col.velocity[:nf] = v
    return col


def _tank(nx, ny, nz):
    return (max(nx + 2, round(3.2 * nx)), max(ny + 2, round(2.2 * ny)), max(nz + 2, round(1.5 * nz)))


def _search_radius(case):
    """About 34 neighbors for uniform points, as 10^6 points at r = 0.02 have; 0.02 for the blobs."""
    if case["points"] == "blobs":
        return 0.02
    return float(np.float32(0.02 * (1e6 / case["n"]) ** (1 / 3)))


def _collection(case, seed):
    if case["kind"] in ("sesph2d", "iisph2d"):
        nx, ny = case["nx"], case["ny"]
        return _flow(scenes.breaking_dam_2d(nx, ny, width=3 * nx, height=max(ny + 20, round(2.4 * ny)), seed=seed),
                     seed, 0.2)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return _flow(scenes.breaking_dam_3d(nx, ny, nz, 1.0, tank=_tank(nx, ny, nz), seed=seed,
                                        layers=case.get("layers", 1)), seed, 0.2)


def _batch_collections(case, seed):
    """The sizes depend on the case alone, the jitter and the noise on the seed too."""
    out = []
    rng = np.random.default_rng(case["count"])
    for i in range(case["count"]):
        f = math.exp(rng.uniform(math.log(case["smallest"]), math.log(case["largest"])))
        nx = max(6, round((f * rng.uniform(0.5, 2.0)) ** (1 / 3)))
        ny = max(6, round(f ** (1 / 3)))
        nz = max(6, round(f / (nx * ny)))
        out.append(_flow(scenes.breaking_dam_3d(nx, ny, nz, 1.0, tank=_tank(nx, ny, nz), seed=seed * 1009 + i),
                         seed * 1009 + i, 0.2))
    return out


def _points(case, seed):
    if case["points"] == "uniform":
        return scenes.ns_points_uniform(case["n"], seed)
    return scenes.ns_points_blobs(case["n"], blobs=64, sigma=0.03, seed=seed)


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _pinned_collection(col):
    return ParticleCollection(**{k: _pinned(getattr(col, k)) for k in ("position", "velocity", "mass", "density", "type")})


def _outputs(n, dim):
    vec, sca = (lambda: _pinned(np.zeros((n, dim), np.float32))), (lambda: _pinned(np.zeros(n, np.float32)))
    return ParticleCollection(position=vec(), velocity=vec(), density=sca(), pressure=sca())


def _configure(s, kind):
    s.parameters.rest_density, s.parameters.gravity, s.parameters.particle_size = 1.0, 9.81, 1.0
    s.timestep_generator.settings.timestep = DT[kind]
    if kind == "sesph2d":
        s.settings.StiffnessK, s.settings.Viscosity = 1000.0, 0.01
    elif kind == "iisph2d":
        s.settings.Viscosity = 0.01
    elif kind == "sesph3d":
        s.settings.StiffnessK, s.settings.Viscosity = 1000.0, 0.01
    else:
        s.settings.viscosity = 0.01


SOLVERS = {"sesph2d": SESPHFluidSolver, "iisph2d": IISPHFluidSolver, "sesph3d": SESPHFluidSolver3D,
           "iisph3d": IISPHFluidSolver3D}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "search":
        s = NeighborhoodSearch(case["search"], _search_radius(case))
        s.data.collection = ParticleCollection(position=_points(case, seed))
        s.initialize()
        room = case["n"] * 40 if case["points"] == "uniform" else int(case["n"] * (20 + case["n"] / 64 * 0.09))
        return dict(case=case, solver=s, offsets=np.zeros(case["n"] + 1, np.int64), indices=np.zeros(room, np.int64))
    if kind == "render":
        s = IISPHFluidSolver3D(search="hashed-3d")
        _configure(s, "iisph3d")
        s.data.collection = _collection(case, seed)
        s.initialize()
        c = (case["nx"] / 2, case["ny"] / 2, case["nz"] / 2)
        eye = (3.0 * case["nx"], 1.4 * case["ny"], 2.2 * case["nz"])
        look = tuple(float(a - b) for a, b in zip(c, eye))
        return dict(case=case, solver=s, eye=eye, look=look, seed=seed % 1000 + 1)
    if kind == "batch":
        cols = _batch_collections(case, seed)
        s = BatchedIISPHFluidSolver3D(cols)
        _configure(s, kind)
        s.settings.single_layer_boundary = True
        s.initialize()
        whole = ParticleCollection(**{k: np.concatenate([getattr(c, k) for c in cols])
                                      for k in ("position", "velocity", "mass", "density", "type")})
        return dict(case=case, solver=s, input=_pinned_collection(whole), out=_outputs(len(whole), 3))
    mode = case["mode"]
    s = SOLVERS[kind](search=case["search"], precision={"fast": "fp32-kahan", "exact": "fp32", "fp64": "fp64"}[mode],
                      reference_order=mode == "exact")
    _configure(s, kind)
    if kind in ("iisph3d", "sesph3d"):
        s.settings.single_layer_boundary = case["layers"] == 1
    s.data.collection = _pinned_collection(_collection(case, seed))
    s.initialize()
    return dict(case=case, solver=s, out=_outputs(len(s.data.collection), s.data.collection.dim))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case, s = state["case"], state["solver"]
    kind = case["kind"]
    if kind == "search":
        s.data.notify_that_data_changed()
        s.find_neighbors()
        off, idx, total = state["offsets"], state["indices"], ctypes.c_int64()
        F.check(F.lib().fs_get_neighbors_csr(s.ctx, off.ctypes.data, None, ctypes.byref(total)))
        if total.value > len(idx):   # a program would make its array larger
            raise MemoryError("more neighbors than the kept array holds")
        F.check(F.lib().fs_get_neighbors_csr(s.ctx, off.ctypes.data, idx.ctypes.data, ctypes.byref(total)))
        return dict(offsets=off, indices=idx)
    if kind == "render":
        radiance, rgba = s.render(state["eye"], state["look"], width=case["width"], height=case["height"],
                                  samples_per_pixel=case["samples"], maximum_recursion_depth=case["depth"],
                                  seed=state["seed"])
        return dict(radiance=radiance, rgba=rgba)
    out = state["out"]
    if kind == "batch":
        F.check(F.lib().fs_upload(s.ctx, ctypes.byref(state["input"].as_fs())))
        stats = s.run(case["steps"])
        iterations = np.array([st.iterations for st in stats], np.int32)
        dt = np.array([st.actual_dt for st in stats], np.float32)
    elif case.get("calls") == "pair":
        tp = Timepoint(desired_time_step=DT[kind])
        s.data.notify_that_data_changed()
        for _ in range(case["steps"]):
            s.execute_neighborhood_search()
            s.execute_simulation_step(tp)
        iterations, dt = np.array([s.last_stats.iterations], np.int32), np.array([tp.actual_time_step], np.float32)
    else:
        s.data.notify_that_data_changed()
        st = s.run(case["steps"])
        iterations, dt = np.array([st.iterations], np.int32), np.array([st.actual_dt], np.float32)
    F.check(F.lib().fs_download(s.ctx, ctypes.byref(out.as_fs())))
    res = {k: getattr(out, k) for k in OUTPUTS}
    res.update(iterations=iterations, dt=dt)
    return res


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(case):
    """(fluid, boundary) particles of a dam."""
    nx, ny = case["nx"], case["ny"]
    if "nz" not in case:
        w, h = 3 * nx, max(ny + 20, round(2.4 * ny))
        return nx * ny, 3 * (w + 6) + 6 * h
    return _counts3(nx, ny, case["nz"], case.get("layers", 1))


def _counts3(nx, ny, nz, layers):
    lx, ly, lz = _tank(nx, ny, nz)
    b = 0
    for k in range(1, layers + 1):
        b += (lx + 2 * k) * (lz + 2 * k) + 2 * (ly + k - 1) * (lz + 2 * k - 2) + 2 * (ly + k - 1) * (lx + 2 * k)
    return nx * ny * nz, b


def _step_work(f, b, steps, iterations, dim, size):
    """Bytes: the collection in (position, velocity, mass, density, type) and the fields out, once; per step the
    search's and the phases' particle fields read and written once (144 bytes for every particle, 120 for every fluid
    particle, 84 more for every iteration of the pressure loop; a real of `size` bytes), without lists. Operations:
    per neighbor pair about 20 for a search's test and 45 for a loop over the neighbors."""
    n = f + b
    pairs = f * (32 if dim == 3 else 20)
    host = n * (8 * dim + 9) + n * (8 * dim + 8)
    per = (144 * n + 216 * f + 84 * f * iterations) * size / 4
    return host + steps * per, steps * pairs * (20 + 45 * (2 + 2 * iterations))


def work(case):
    kind = case["kind"]
    if kind == "search":
        per = 34 if case["points"] == "uniform" else 1 + case["n"] / 64 * 0.028
        return dict(bytes=case["n"] * (12.0 + 8 + 8 * per), flops=case["n"] * per * 6.5 * 8.0)
    if kind == "render":
        # the march points whose neighborhood is not empty: about a quarter of the box's depth for each ray
        rays = case["width"] * case["height"] * case["samples"] * 3.0
        f, b = _counts(case)
        return dict(bytes=(f + b) * 17.0 + case["width"] * case["height"] * 16.0, flops=rays * 60 * 30 * 40.0)
    iterations = {"sesph2d": 0, "sesph3d": 0, "iisph2d": 2, "iisph3d": 6, "batch": 6}[kind]
    if kind == "batch":
        rng = np.random.default_rng(case["count"])
        f = b = 0
        for _ in range(case["count"]):
            q = math.exp(rng.uniform(math.log(case["smallest"]), math.log(case["largest"])))
            nx = max(6, round((q * rng.uniform(0.5, 2.0)) ** (1 / 3)))
            ny = max(6, round(q ** (1 / 3)))
            a = _counts3(nx, ny, max(6, round(q / (nx * ny))), 1)
            f, b = f + a[0], b + a[1]
        byts, flops = _step_work(f, b, case["steps"], iterations, 3, 4)
    else:
        f, b = _counts(case)
        byts, flops = _step_work(f, b, case["steps"], iterations, 3 if "nz" in case else 2,
                                 8 if case["mode"] == "fp64" else 4)
    return dict(bytes=float(byts), flops=float(flops))


# ---------------------------------------------------------------------------
# the same passes in 64 bits, in plain torch
# ---------------------------------------------------------------------------
class _Exact:
    """One dam's solver in 64 bits. The settings are the 32-bit values that the solver is given."""

    def __init__(self, kind, col, single_layer, serial_density):
        f = lambda v: float(np.float32(v))
        self.kind, self.dim = kind, col.position.shape[1]
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)
        self.x, self.v = t(col.position).double(), t(col.velocity).double()
        self.m, self.rho = t(col.mass).double(), t(col.density).double()
        self.fluid = t(col.type) == 0
        n = len(col.position)
        self.p, self.acc = torch.zeros(n, device=self.dev).double(), torch.zeros_like(self.x)
        self.h, self.r = 1.0, 2.0
        self.alpha = 1 / (4 * math.pi) if self.dim == 3 else 5 / (14 * math.pi)
        self.nu2, self.eps, self.gravity = 2 * f(0.01), f(0.01), f(9.81)
        self.gamma, self.omega, self.gamma1, self.stiffness = f(0.7), f(0.5), f(1.1), 1000.0
        self.max_error, self.lambda_v, self.lambda_a = f(0.001), f(0.4), f(0.25)
        self.single, self.serial = single_layer, serial_density
        self.dt0 = f(DT[kind])
        self.dt, self.iterations = self.dt0, 0

    def pairs(self):
        """(i, j): fluid owner i, every j within the radius, i itself included."""
        c = torch.floor(self.x / self.r).long()
        c = c - c.min(0).values + 1
        dims = c.max(0).values + 2
        lin = c[:, 0]
        for a in range(1, self.dim):
            lin = lin * dims[a] + c[:, a]
        order = torch.argsort(lin)
        keys = lin[order]
        own = torch.nonzero(self.fluid).flatten()
        strides = [1]
        for a in range(self.dim - 1, 0, -1):
            strides.insert(0, strides[0] * int(dims[a]))
        ii, jj = [], []
        for k in range(3 ** self.dim):
            shift = sum((k // 3 ** a % 3 - 1) * strides[a] for a in range(self.dim))
            at = lin[own] + shift
            lo, hi = torch.searchsorted(keys, at), torch.searchsorted(keys, at, right=True)
            cnt = hi - lo
            i = torch.repeat_interleave(own, cnt)
            first = torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt - lo, cnt)
            j = order[torch.arange(i.numel(), device=self.dev) - first]
            near = ((self.x[i] - self.x[j]) ** 2).sum(1) <= self.r * self.r
            ii.append(i[near])
            jj.append(j[near])
        return torch.cat(ii), torch.cat(jj)

    def spline(self, d):
        q = d.norm(dim=1) / self.h
        a, b = (2 - q).clamp(min=0), (1 - q).clamp(min=0)
        w = self.alpha * (a ** 3 - 4 * b ** 3)
        f = self.alpha * (-3 * a ** 2 + 12 * b ** 2) / (q * self.h * self.h).clamp(min=1e-30)
        return w, torch.where((q > 1e-7)[:, None], f[:, None] * d * self.h, torch.zeros_like(d))

    def sum(self, i, val):
        out = torch.zeros((len(self.x),) + tuple(val.shape[1:]), dtype=torch.float64, device=self.dev)
        return out.index_add_(0, i, val)

    def cfl(self, a2, v2):
        ma, mv = math.sqrt(a2), math.sqrt(v2)
        ta = math.sqrt(1.0 / ma) * self.lambda_a if ma > 0 else self.dt0
        tv = 1.0 / mv * self.lambda_v if mv > 0 else self.dt0
        return min(max(min(ta, tv), 1e-6), self.dt0)

    def step(self):
        dot = lambda a, b: (a * b).sum(1)
        i, j = self.pairs()
        fl = self.fluid[j]
        d = self.x[i] - self.x[j]
        w, g = self.spline(d)
        m = self.m[j]
        three, iisph = self.dim == 3, self.kind.startswith("iisph") or self.kind == "batch"
        wm = torch.where(fl, m, m * self.gamma1) if three and self.single else m
        new = torch.where(self.fluid, self.sum(i, wm * w), self.rho)
        if not iisph:
            rj = new[j]
        elif self.serial:   # the serial loop overwrites the densities that it reads
            rj = torch.where(fl & (j < i), new[j], self.rho[j])
        else:
            rj = self.rho[j]
        vij = self.v[i] - self.v[j]
        term = torch.where(rj == 0, torch.zeros_like(rj), m / rj * dot(vij, d) / (dot(d, d) + self.eps))
        down = torch.zeros_like(self.x)
        down[:, 1] = -self.gravity
        npa = torch.where(self.fluid[:, None], self.nu2 * self.sum(i, term[:, None] * g) + down, torch.zeros_like(self.x))
        self.rho = new
        if not iisph:
            self.p = torch.where(self.fluid, (self.stiffness * (new - 1)).clamp(min=0), self.p)
            pdd = self.p / new ** 2
            g2 = self.gamma1 if three and self.single else 1.0
            c = torch.where(fl, -m * (pdd[i] + pdd[j]), -self.m[i] * 2 * pdd[i] * g2)
            self.acc = torch.where(self.fluid[:, None], self.sum(i, c[:, None] * g) + npa, self.acc)
            if three:
                v = self.v + self.dt0 * self.acc
                self.dt = self.cfl(float(dot(self.acc, self.acc).max()), float(dot(v, v).max()))
            self.v = self.v + self.dt * self.acc
            self.x = self.x + self.dt * self.v
            return
        dt = self.dt0
        vs = self.v + dt * npa
        if three:
            self.p = torch.zeros_like(self.p)
            dv = torch.where(fl[:, None], vs[i] - vs[j], vs[i])
            wb = 2 * self.gamma if self.single else 2.0
            pb = wb
        else:
            self.p = torch.where(self.fluid, torch.zeros_like(self.p), self.p)
            dv = vs[i] - vs[j]
            wb = pb = 2 * self.gamma
        source = (1 - new) - dt * self.sum(i, m * dot(dv, g))
        inner = -self.sum(i, torch.where(fl, m, wb * m)[:, None] * g)
        diag = self.sum(i, m * dot(inner[i], g) - torch.where(fl, m * self.m[i] * dot(g, g), torch.zeros_like(m))) * dt * dt
        has = self.fluid & (diag.abs() > 1.19209290e-07)
        safe = torch.where(has, diag, torch.ones_like(diag))
        it = 0
        while True:
            c = torch.where(fl, m * (self.p[i] + self.p[j]), pb * m * self.p[i])
            a = -self.sum(i, c[:, None] * g)
            self.acc = torch.where(self.fluid[:, None], a, self.acc)
            da = torch.where(fl[:, None], self.acc[i] - self.acc[j], self.acc[i])
            ap = self.sum(i, m * dot(da, g)) * dt * dt
            p = (self.p + self.omega * (source - ap) / safe).clamp(min=0)
            self.p = torch.where(self.fluid, torch.where(has, p, torch.zeros_like(p)), self.p)
            err = torch.where(self.p > 1.19209290e-07, (source - ap).abs(), torch.zeros_like(ap))[has]
            avg = float(err.mean()) if err.numel() else 0.0
            it += 1
            if it >= 100 or it >= 2 and (avg <= self.max_error if three else float(int(avg)) <= self.max_error):
                break
        self.iterations = it
        if three:
            v = (vs + dt * self.acc)[self.fluid]
            a = self.acc[self.fluid]
            self.dt = self.cfl(float(dot(a, a).max()), float(dot(v, v).max()))
        self.v = (vs - dt * npa) + self.dt * npa + self.dt * self.acc
        self.x = self.x + self.dt * self.v

    def result(self, steps):
        for _ in range(steps):
            self.step()
        c = lambda a: a.cpu()
        return dict(position=c(self.x), velocity=c(self.v), density=c(self.rho), pressure=c(self.p), iterations=np.array([self.iterations], np.int32), dt=np.array([self.dt]))


def exact(case, seed):
    """Neighbor lists are whole numbers, and a path-traced image is a sample, whose rays part at the last bit of a
    density: neither has a value in 64 bits."""
    kind = case["kind"]
    if kind in ("search", "render"):
        return None
    if kind == "batch":
        parts = [_Exact("iisph3d", c, True, False).result(case["steps"]) for c in _batch_collections(case, seed)]
        return {k: np.concatenate([np.asarray(p[k]) for p in parts]) for k in parts[0]}
    serial = case["mode"] == "exact" and kind.startswith("iisph")
    e = _Exact(kind, _collection(case, seed), case.get("layers") == 1, serial)
    return e.result(case["steps"])
