"""Exports that have nothing to export: the solver's lists after a search that a
NaN ended, which has built none."""
import numpy as np
import pytest

from fluidsolver_b200._lib import FS_ERR_NAN, FS_ERR_STATE, FluidSolverError
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
