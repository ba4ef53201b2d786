"""Contexts of different list capacities side by side: what one of them needs
in shared memory does not depend on which was created last. And the capacities
that the fast mode refuses."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200._lib import FluidSolverError
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


def solver(capacity, n=4000):
    s = make_solver("iisph-3d", "hashed-3d", [0.001, 2, 9, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                    precision="fp32-kahan", neighbor_capacity=capacity)
    s.data.collection = dam(n, 3)
    s.initialize()
    return s


@pytest.mark.parametrize("capacity", [64, 256, 384, 512])
@pytest.mark.parametrize("n", [4000, 80000])
def test_a_smaller_context_created_later(capacity, n):
    alone = solver(capacity, n)
    alone.step()
    want = alone.collection()
    alone.close()
    a = solver(capacity, n)
    b = solver(0)
    a.step()
    b.step()
    got = a.collection()
    for f in ("position", "velocity", "density", "pressure"):
        assert bits_equal(getattr(got, f), getattr(want, f)), f
    a.close()
    b.close()


@pytest.mark.parametrize("capacity", [520, 704, 712])
def test_refused_capacities(capacity):
    with pytest.raises(FluidSolverError):
        solver(capacity)
