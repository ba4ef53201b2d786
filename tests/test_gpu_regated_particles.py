"""Uploads of the same particles with some of them switched between boundary
and inactive (a gate that opens): the particle and fluid counts stay, and the
steps captured for one upload must not be replayed for the next, whose
structure holds other particles. Against contexts of their own, bit for bit."""
import ctypes

import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import _lib as F
from fluidsolver_b200 import scenes
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


def dam(inactive):
    """A dam that touches every wall, with `inactive` of its boundary particles switched off, none of the outermost
    ones (so that the box and the grid stay)."""
    c = scenes.breaking_dam_3d(20, 20, 20, 1.0, tank=(21, 21, 21), seed=5).collection
    typ = c.type.copy()
    lo, hi = c.position.min(0), c.position.max(0)
    inner = np.flatnonzero((typ == 1) & (((c.position > lo + 2) & (c.position < hi - 2)).sum(1) >= 2))
    typ[inner[:inactive]] = 2
    assert (typ == 2).sum() == inactive
    return ParticleCollection(position=c.position, velocity=np.zeros_like(c.position), mass=c.mass,
                              density=np.ones(len(c), np.float32), type=typ)


@pytest.mark.parametrize("counts", [(0, 1300, 0), (1300, 200, 1300), (1100, 1000, 1100)])
@pytest.mark.parametrize("precision", ["fp32-kahan", "fp32"])
def test_runs_after_each_upload(counts, precision):
    make = lambda: make_solver("iisph-3d", "hashed-3d", [0.001, 2, 10, 0.5, 0.7, 0.01, 1.0, 1.1],  # noqa: E731
                               (0.005, 0.4, 0.25), precision=precision)
    kept = make()
    kept.data.collection = dam(counts[0])
    kept.initialize()
    for inactive in counts:
        col = dam(inactive)
        F.check(F.lib().fs_upload(kept.ctx, ctypes.byref(col.as_fs())))
        fresh = make()
        fresh.data.collection = col
        a, b = kept.run(6), fresh.run(6)   # (the buffers are where they were after six)
        assert (a.iterations, a.max_neighbors) == (b.iterations, b.max_neighbors), inactive
        x, y = kept.collection(), fresh.collection()
        for f in ("position", "velocity", "density", "pressure"):
            assert bits_equal(getattr(x, f), getattr(y, f)), (inactive, f)
        fresh.close()
    kept.close()
