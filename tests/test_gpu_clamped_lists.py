"""Solver lists in a grid that is smaller than the particles' box (two particles
far away on either side): owners whose neighborhood lies in its border cells,
among all the particles that are clamped into them, and owners on both sides of
the edge. The bit-exact steps against the oracle, which they follow only with
the right lists in the right order; the lists' members against the contract's."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import scenes
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu

SETTINGS = {"sesph-2d": [1000.0, 0.01], "iisph-3d": [0.001, 2, 20, 0.5, 0.7, 0.01, 1.0, 1.1]}


def grid_dims(dim, lo, hi, max_cells=1 << 22):
    """The grid that an upload chooses for a box of cells."""
    ext = [1, 1, 1]
    for a in range(dim):
        e = hi[a] - lo[a] + 1
        ext[a] = min(1 << 20, e + 2 * max(2, e // 16))
    while ext[0] * ext[1] * ext[2] > max_cells:
        a = 0 if ext[0] >= ext[1] and ext[0] >= ext[2] else (1 if ext[1] >= ext[2] else 2)
        ext[a] = max(1, ext[a] * 3 // 4)
    return ext


def scene(solver, where):
    """A small dam with a far boundary particle on either side, so that the grid, which begins at the
    box's lower corner, ends before the dam ("corner"), or within it along x ("edge")."""
    dim = 2 if solver.endswith("2d") else 3
    if dim == 2:
        c, far = scenes.breaking_dam_2d(24, 24, width=40, height=40, seed=3).collection, 20000.0
    else:
        c, far = scenes.breaking_dam_3d(9, 9, 9, 1.0, tank=(16, 12, 12), seed=3).collection, 1500.0
    for near in (far, *np.arange(20.0, far, 7.0)):
        lo = np.full(dim, -far, np.float32)
        lo[0] = -near
        hi = np.full(dim, far, np.float32)
        d = grid_dims(dim, np.floor(lo / 2).astype(int), np.floor(hi / 2).astype(int))
        end = 2 * (np.floor(lo[0] / 2) + d[0])   # where the grid ends along x
        if where == "corner" and end < -10 or where == "edge" and 5 < end < 9:
            break
    else:
        raise AssertionError("no such grid")
    pos = np.concatenate([c.position, lo[None], hi[None]]).astype(np.float32)
    n = len(pos)
    rng = np.random.default_rng(5)
    return ParticleCollection(position=pos, velocity=rng.normal(0, 0.05, pos.shape).astype(np.float32),
                              mass=np.ones(n, np.float32), density=np.ones(n, np.float32),
                              type=np.concatenate([c.type, [1, 1]]).astype(np.uint8))


@pytest.mark.parametrize("where", ["corner", "edge"])
@pytest.mark.parametrize("solver,search", [("sesph-2d", "hashed-2d"), ("sesph-2d", "quadratic-2d"),
                                           ("iisph-3d", "hashed-3d"), ("iisph-3d", "quadratic-3d")])
def test_bit_exact_steps(c_oracle, solver, search, where):
    col = scene(solver, where)
    dt = 0.001
    s = make_solver(solver, search, SETTINGS[solver], (dt, 0.4, 0.25), precision="fp32", reference_order=True)
    s.data.collection = col
    ref = c_oracle.State(col)
    kw = dict(single_layer=False) if solver == "sesph-2d" else dict(max_it=20)
    ref.run(c_oracle.config(solver, search, timestep=dt, **kw), 3)
    s.run(3)
    out = s.collection()
    for f in ("position", "velocity", "density", "pressure"):
        assert bits_equal(getattr(out, f), getattr(ref, f)), f
    s.close()


@pytest.mark.parametrize("where", ["corner", "edge"])
@pytest.mark.parametrize("precision,reference_order", [("fp32", False), ("fp64", False), ("fp32", True), ("fp32-kahan", False)])
@pytest.mark.parametrize("solver,search", [("sesph-2d", "hashed-2d"), ("iisph-3d", "hashed-3d")])
def test_members(solver, search, precision, reference_order, where):
    col = scene(solver, where)
    s = make_solver(solver, search, SETTINGS[solver], (0.001, 0.4, 0.25), precision=precision,
                    reference_order=reference_order)
    s.data.collection = col
    s.execute_neighborhood_search()
    off, idx = s.solver_lists()
    want_off, want = s.neighbor_lists()
    fluid = np.flatnonzero(col.type == 0)
    assert np.array_equal(np.diff(off)[fluid], np.diff(want_off)[fluid])
    for k in fluid:
        assert np.array_equal(idx[off[k]:off[k + 1]], want[want_off[k]:want_off[k + 1]])
    s.close()
