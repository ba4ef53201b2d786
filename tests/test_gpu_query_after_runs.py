"""Position queries walk the cells of the last search, and a step is one: after a
new upload and steps that replay a captured graph as well as after the first."""
import numpy as np
import pytest

from fluidsolver_b200._lib import FS_ERR_STATE, FluidSolverError
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32-kahan", "fp32"])
def test_queries_after_replayed_steps(precision):
    s = make_solver("iisph-3d", "hashed-3d", [0.001, 2, 9, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                    precision=precision)
    s.data.collection = dam(3000, 5)
    found = []
    for _ in range(3):
        s.data.notify_that_data_changed()
        s.initialize()
        with pytest.raises(FluidSolverError) as e:
            s.get_neighbors_of_position([4.0, 4.0, 4.0])
        assert e.value.status == FS_ERR_STATE
        s.run(6)
        found.append(s.get_neighbors_of_position([4.0, 4.0, 4.0]))
    assert len(found[0]) > 0
    assert all(np.array_equal(f, found[0]) for f in found)
    s.close()
