"""Steps queued behind one that an error has ended: all positions become NaN in
the first step, and the later searches put all particles into one cell. The run
returns FS_ERR_NAN, and the state keeps every particle (the fields that no
phase has touched come back in host order)."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import scenes
from fluidsolver_b200._lib import FS_ERR_NAN, FluidSolverError
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,search,kw", [
    ("iisph-3d", "hashed-3d", dict(precision="fp32-kahan")), ("iisph-3d", "hashed-3d", dict(precision="fp32", reference_order=True)),
    ("sesph-3d", "hashed-3d", dict(precision="fp32-kahan")), ("sesph-2d", "hashed-2d", dict(precision="fp32", reference_order=True)),
    ("sesph-2d", "quadratic-2d", dict(precision="fp32-kahan"))])
@pytest.mark.parametrize("steps", [2, 9])
def test_all_positions_nan(solver, search, kw, steps):
    if solver.endswith("2d"):
        col, settings = scenes.breaking_dam_2d(60, 60, width=140, height=90, seed=3).collection, [1000.0, 0.01]
    else:
        col = dam(30000, 5)
        settings = [0.001, 2, 9, 0.5, 0.7, 0.01, 1.0, 1.1] if solver == "iisph-3d" else [1000.0, 0.01, 1, 1.1, 1.1]
    n = len(col)
    mass = np.random.default_rng(4).uniform(0.9, 1.1, n).astype(np.float32)
    s = make_solver(solver, search, settings, (0.001, 0.4, 0.25), **kw)
    s.data.collection = ParticleCollection(position=col.position, velocity=np.full_like(col.position, np.nan), mass=mass,
                                           density=np.ones(n, np.float32), type=col.type)
    with pytest.raises(FluidSolverError) as e:
        s.run(steps)
    assert e.value.status == FS_ERR_NAN
    out = s.collection()
    assert bits_equal(out.mass, mass) and bits_equal(out.type, col.type)
    assert np.isnan(out.position).all()
    s.data.collection.velocity = np.zeros_like(col.position)   # and the context goes on with other particles
    s.data.notify_that_data_changed()
    assert s.run(2).status == 0
    s.close()
