"""The ray march's shared evaluation (a warp per ray, several march points and
one list of candidates at a time) against a plain serial march over all
particles, at the cases where its paths differ: sparse particles far apart
(empty stretches and the map of occupied neighborhoods), more candidates
around a point than one window of the list holds (128), directions longer than
one (points cells apart, evaluated one by one), both particle regions, and the
reference-order mode's single region."""
import numpy as np
import pytest

from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


def serial_march(pos, mass, bnd, o, d, iso, lo, hi):
    """First crossing of the density along o + (step t) d in double, or None; the smallest distance
    of a visited density, or density difference, to the decision it takes part in."""
    def volume(x):
        q = np.linalg.norm(x - pos, axis=1)
        a, b = np.clip(2 - q, 0, None), np.clip(1 - q, 0, None)
        c = np.where(q <= 2, mass * (a ** 3 - 4 * b ** 3) / (4 * np.pi), 0)
        return c[~bnd].sum(), c[bnd].sum()

    def state(v):
        return 0 if v[0] + v[1] < iso else (1 if v[0] > v[1] else 2)

    last, within, near = volume(o + 0.25 * d), False, np.inf
    for t in range(1, 4000):
        p = o + 0.5 * t * d
        if np.any(p < lo) or np.any(p > hi):
            if within:
                break
            continue
        within = True
        cur = volume(p)
        near = min(near, abs(cur[0] + cur[1] - iso))
        a, b = state(last), state(cur)
        if a != b and a != 2:
            return (0 if b == 1 else 2) if a == 0 else (1 if b == 0 else 2), 0.5 * t, near
        last = cur
    return None, -1.0, near


@pytest.mark.parametrize("scale,dense,exact", [(1.0, False, False), (1.0, True, False), (7.3, False, False),
                                               (1.0, False, True)])
def test_march_matches_a_serial_march(scale, dense, exact):
    rng = np.random.default_rng(5)
    spacing = 0.4 if dense else 1.0   # 0.4: about 500 particles within the radius, 3,400 in the 27 cells
    g = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3) * spacing
    far = rng.uniform(-25, 25, (30, 3))
    pos = np.concatenate([g, g + [18.0, 3.0, -9.0], far]).astype(np.float32)
    bnd = np.concatenate([np.zeros(216, bool), np.ones(216, bool), np.zeros(30, bool)])
    mass = np.full(len(pos), spacing ** 3, np.float32)
    s = make_solver("iisph-3d", "hashed-3d", [0.001, 2, 100, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                    precision="fp32" if exact else "fp32-kahan", reference_order=exact)
    s.data.collection = ParticleCollection(position=pos, velocity=np.zeros_like(pos), mass=mass,
                                           density=np.ones(len(pos), np.float32), type=bnd.astype(np.uint8))
    target = np.concatenate([pos[rng.integers(0, 216, 40)], pos[rng.integers(216, 432, 40)], pos[-20:]])
    o = (target + rng.normal(0, 1, target.shape) * 30).astype(np.float32)
    d = target - o
    d = (scale * d / np.linalg.norm(d, axis=1)[:, None]).astype(np.float32)
    got = s.trace_rays(o, d)
    s.close()
    lo, hi = pos.min(0) - 2, pos.max(0) + 2
    hits = 0
    for i in range(len(o)):
        kind, length, near = serial_march(pos.astype(np.float64), mass.astype(np.float64), bnd, o[i].astype(np.float64),
                                          d[i].astype(np.float64), np.float32(0.8), lo, hi)
        if near < 1e-4:
            continue   # a density within rounding of the surface density
        assert got["hit"][i] == (-1 if kind is None else kind), i
        assert got["length"][i] == np.float32(length), i
        hits += kind is not None
    assert hits > 20 if scale == 1.0 else True
