"""Uploads that are refused after their particles were counted: the next upload
counts from the start, and the state of the last one that succeeded stays as
it was. The scenes of a batch whose grids together exceed 2^30 cells (one far
particle in each of 360 scenes) are refused."""
import ctypes

import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import _lib as F
from fluidsolver_b200.solver import BatchedIISPHFluidSolver3D, ParticleCollection

pytestmark = pytest.mark.gpu
SCENES, SIDE = 360, 3


def batch(seed, far=False):
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(SIDE)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)
    cols = []
    for i in range(SCENES):
        p = (g + rng.uniform(-0.05, 0.05, g.shape)).astype(np.float32)
        if far:
            p[-1] = 3000.0 + i
        typ = (np.arange(len(p)) % 5 == seed % 5).astype(np.uint8)
        cols.append(ParticleCollection(position=p, velocity=rng.normal(0, 0.1, p.shape).astype(np.float32),
                                       mass=np.ones(len(p), np.float32), density=np.ones(len(p), np.float32), type=typ))
    return cols


def whole(cols):
    return ParticleCollection(**{f: np.ascontiguousarray(np.concatenate([getattr(c, f) for c in cols]))
                                 for f in ("position", "velocity", "mass", "density", "type")})


def solver(cols):
    s = BatchedIISPHFluidSolver3D(cols)
    s.parameters.rest_density, s.parameters.gravity, s.parameters.particle_size = 1.0, 9.81, 1.0
    s.settings.viscosity = 0.01
    s.timestep_generator.settings.timestep = 0.005
    s.initialize()
    return s


def upload(s, cols):
    col = whole(cols)
    return F.lib().fs_upload(s.ctx, ctypes.byref(col.as_fs()))


def state(s):
    c = s.collections()
    return {f: np.concatenate([getattr(x, f) for x in c]) for f in ("position", "velocity", "density", "pressure")}


@pytest.mark.parametrize("then_upload", [True, False])
def test_after_grids_that_are_too_large(then_upload):
    first, second = batch(1), batch(2)
    s = solver(first)
    for _ in range(2):
        assert upload(s, batch(3, far=True)) == F.FS_ERR_INVALID
    if then_upload:
        F.check(upload(s, second))
    fresh = solver(second if then_upload else first)
    a = [(x.iterations, x.actual_dt) for x in s.run(3)]
    b = [(x.iterations, x.actual_dt) for x in fresh.run(3)]
    assert a == b
    sa, sb = state(s), state(fresh)
    for f in sa:
        assert bits_equal(sa[f], sb[f]), f
    s.close()
    fresh.close()
