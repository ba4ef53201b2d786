"""Lists that would have to grow beyond the device's memory: 250,000 particles
within one radius ask for 250 GB. Every step of them fails, and the context goes
on with other particles."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200._lib import FluidSolverError
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu
SIDE = 63


def particles(spacing):
    g = np.stack(np.meshgrid(*[np.arange(SIDE)] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = (g * spacing + np.random.default_rng(2).uniform(-0.02, 0.02, g.shape) * spacing).astype(np.float32)
    return ParticleCollection(position=p, velocity=np.zeros_like(p), mass=np.ones(len(p), np.float32),
                              density=np.ones(len(p), np.float32), type=np.zeros(len(p), np.uint8))


def solver(spacing):
    s = make_solver("sesph-3d", "hashed-3d", [1000.0, 0.01, 1, 1.1, 1.1], (0.001, 0.4, 0.25), precision="fp32")
    s.data.collection = particles(spacing)
    return s


def test_steps_after_lists_that_could_not_grow():
    s, other = solver(0.01), solver(1.0)
    for call in (s.step, s.step, s.execute_neighborhood_search, lambda: s.run(3)):
        with pytest.raises(FluidSolverError):
            call()
    s.data.collection = particles(1.0)
    s.data.notify_that_data_changed()
    s.run(3)
    other.run(3)
    a, b = s.collection(), other.collection()
    for f in ("position", "velocity", "density", "pressure"):
        assert bits_equal(getattr(a, f), getattr(b, f)), f
    s.close()
    other.close()
