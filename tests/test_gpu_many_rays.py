"""Rays beyond 32,768 in a call are marched by a thread each instead of a warp: the
same hits, points, normals and lengths, bit for bit, as the same rays in calls
of fewer. Rays from outside, from within the fluid, along the axes, beside the
box and away from it; a grid smaller than the particles' box."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu
LINE = 32768


def rays(n, side):
    rng = np.random.default_rng(n)
    o = rng.uniform(-side, 3 * side, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    o[::3] = rng.uniform(0, side, (len(o[::3]), 3))                          # within the fluid
    d[1::3] = rng.uniform(0, side, (len(d[1::3]), 3)) - o[1::3]              # into it
    axis = np.arange(0, n, 7)
    d[axis] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, len(axis))] * rng.choice([-1, 1], (len(axis), 1))
    return o, (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


@pytest.mark.parametrize("precision,reference_order,stray,n", [
    ("fp32-kahan", False, False, LINE + 1), ("fp32-kahan", False, False, 3 * LINE - 17), ("fp64", False, False, LINE + 1),
    ("fp32", True, False, LINE + 1), ("fp32-kahan", False, True, LINE + 1)])
def test_many_rays_are_the_rays_in_smaller_calls(precision, reference_order, stray, n):
    s = make_solver("iisph-3d", "hashed-3d", [0.001, 2, 9, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                    precision=precision, reference_order=reference_order)
    col = dam(100 if stray else 4000, 5)
    if stray:   # two particles so far away that the grid cannot hold the box
        p = col.position.copy()
        p[-1], p[-2] = 700.0, (-600.0, 500.0, -400.0)
        col = ParticleCollection(position=p, velocity=col.velocity, mass=col.mass, density=col.density, type=col.type)
    s.data.collection = col
    o, d = rays(n, 5 if stray else 16)
    a = s.trace_rays(o, d)
    parts = [s.trace_rays(o[i:i + LINE], d[i:i + LINE]) for i in range(0, n, LINE)]
    assert (a["hit"] >= 0).sum() > n / 20 and (a["hit"] == -1).sum() > n / 20
    for f in a:
        b = np.concatenate([p[f] for p in parts])
        assert bits_equal(a[f], b) or np.array_equal(np.isnan(a[f]), np.isnan(b)) and np.array_equal(
            np.nan_to_num(a[f]), np.nan_to_num(b)), f
    s.close()
