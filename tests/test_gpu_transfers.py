"""Uploads and downloads: what was uploaded comes back bit for bit (nothing is
computed, so there is no tolerance), below and above 4 MB, where a download's
copies run under its scatter; for all fields and for a few; after an upload of
another size; after a refused one."""
import ctypes

import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import _lib as F
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu

IISPH = [0.001, 2, 100, 0.5, 0.7, 0.01, 1.0, 1.1]
FIELDS = ("position", "velocity", "acceleration", "external", "mass", "density", "pressure", "type", "tag")


def particles(n, seed):
    rng = np.random.default_rng(seed)
    side = max(1.0, n ** (1 / 3))
    vec = lambda: rng.normal(size=(n, 3)).astype(np.float32)  # noqa: E731
    return ParticleCollection(
        position=rng.uniform(0, side, (n, 3)).astype(np.float32), velocity=vec(), acceleration=vec(), external=vec(),
        mass=rng.uniform(0.5, 1.5, n).astype(np.float32), density=rng.uniform(0.5, 1.5, n).astype(np.float32),
        pressure=rng.uniform(0, 1, n).astype(np.float32), type=rng.integers(0, 3, n).astype(np.uint8),
        tag=np.arange(n, dtype=np.uint32))


def empty(n, fields):
    like = particles(1, 0)
    return ParticleCollection(**{f: np.zeros((n,) + getattr(like, f).shape[1:], getattr(like, f).dtype) for f in fields})


@pytest.mark.parametrize("precision", ["fp32-kahan", "fp64"])
def test_round_trips(precision):
    s = make_solver("iisph-3d", "hashed-3d", IISPH, (0.005, 0.4, 0.25), precision=precision)
    s.data.collection = particles(200000, 1)
    s.initialize()
    for n in (200000, 1, 33, 40000, 70000, 129, 200000):
        col = particles(n, n)
        F.check(F.lib().fs_upload(s.ctx, ctypes.byref(col.as_fs())))
        for fields in (FIELDS, ("position",), ("position", "pressure"), ("type", "position", "velocity", "density")):
            out = empty(n, fields)
            F.check(F.lib().fs_download(s.ctx, ctypes.byref(out.as_fs())))
            for f in fields:
                assert bits_equal(getattr(out, f), getattr(col, f)), (n, fields, f)
    s.close()


def test_upload_after_a_refused_one():
    s = make_solver("iisph-3d", "hashed-3d", IISPH, (0.005, 0.4, 0.25))
    s.data.collection = particles(5000, 2)
    s.initialize()
    bad = particles(5000, 3)
    bad.type[4999] = 7
    assert F.lib().fs_upload(s.ctx, ctypes.byref(bad.as_fs())) == F.FS_ERR_INVALID
    good = particles(5000, 4)
    F.check(F.lib().fs_upload(s.ctx, ctypes.byref(good.as_fs())))
    out = empty(5000, FIELDS)
    F.check(F.lib().fs_download(s.ctx, ctypes.byref(out.as_fs())))
    for f in FIELDS:
        assert bits_equal(getattr(out, f), getattr(good, f)), f
    s.close()
