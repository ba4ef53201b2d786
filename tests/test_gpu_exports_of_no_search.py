"""Exports that have nothing to export: the solver's lists after a search that a
NaN ended, which has built none, and the contract's lists before a search."""
import numpy as np
import pytest

from fluidsolver_b200 import NeighborhoodSearch, scenes
from fluidsolver_b200._lib import FS_ERR_NAN, FS_ERR_STATE, FluidSolverError
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


def refused(call, status):
    with pytest.raises(FluidSolverError) as e:
        call()
    assert e.value.status == status


def solver(precision, n=3000):
    s = make_solver("iisph-3d", "hashed-3d", [0.001, 2, 9, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                    precision=precision)
    s.data.collection = dam(n, 5)
    return s


@pytest.mark.parametrize("precision", ["fp32-kahan", "fp32"])
def test_solver_lists_after_a_nan(precision):
    s = solver(precision)
    good = s.data.collection.position.copy()
    s.data.collection.position[7] = np.nan
    refused(s.execute_neighborhood_search, FS_ERR_NAN)
    refused(s.solver_lists, FS_ERR_STATE)
    s.data.collection.position[7] = good[7]
    s.data.notify_that_data_changed()
    s.execute_neighborhood_search()
    off, idx = s.solver_lists()
    assert off[-1] == len(idx) > 0
    s.close()


@pytest.mark.parametrize("kind", ["iisph-3d", "sesph-2d", "compact", "one kernel"])
def test_neighbor_lists_before_a_search(kind):
    """After a new upload too: the tables still hold the particles before it."""
    if kind == "compact":
        s = NeighborhoodSearch("compact-hashing-2d", 2.0)
    elif kind == "iisph-3d":
        s = solver("fp32-kahan")
    else:
        s = make_solver("sesph-2d", "hashed-2d", [1000.0, 0.01], (0.001, 0.4, 0.25),
                        one_kernel_steps=kind == "one kernel")
    if kind == "compact":
        s.data.collection = ParticleCollection(position=np.arange(40, dtype=np.float32).reshape(20, 2))
        search = s.find_neighbors
    else:
        if kind != "iisph-3d":
            s.data.collection = scenes.breaking_dam_2d(20, 20, width=50, height=40, seed=3).collection
        search = s.step
    for _ in range(2):
        s.data.notify_that_data_changed()
        s.initialize()
        refused(s.neighbor_lists, FS_ERR_STATE)
        search()
        off, idx = s.neighbor_lists()
        assert off[-1] == len(idx) > 0
    s.close()
