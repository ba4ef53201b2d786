"""A NaN position in a context's very first search, in the modes that sort every
list by host index afterwards: the lists have never been written then, so there
is nothing to sort. Below and above the size of one thread per owner, and in
the small-scene kernel."""
import numpy as np
import pytest

from fluidsolver_b200 import scenes
from fluidsolver_b200._lib import FS_ERR_NAN, FluidSolverError
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,search,size,kw", [
    ("sesph-2d", "quadratic-2d", (40, 40), {}), ("sesph-2d", "quadratic-2d", (40, 40), dict(one_kernel_steps=True)),
    ("sesph-2d", "quadratic-2d", (364, 361), {}), ("iisph-2d", "quadratic-2d", (30, 40), dict(one_kernel_steps=True)),
    ("iisph-3d", "quadratic-3d", 3000, {}), ("iisph-3d", "quadratic-3d", 98400, {})])
def test_nan_in_the_first_search(solver, search, size, kw):
    settings = {"sesph-2d": [1000.0, 0.01], "iisph-2d": [0.001, 2, 9, 0.5, 0.7, 0.01],
                "iisph-3d": [0.001, 2, 9, 0.5, 0.7, 0.01, 1.0, 1.1]}[solver]
    col = dam(size, 5) if solver == "iisph-3d" else \
        scenes.breaking_dam_2d(*size, width=2 * size[0], height=size[1] + 20, seed=3).collection
    good = col.position.copy()
    col.position[5] = np.nan
    s = make_solver(solver, search, settings, (0.001, 0.4, 0.25), precision="fp32", reference_order=True, **kw)
    s.data.collection = col
    for call in (s.step, s.execute_neighborhood_search, lambda: s.run(3)):
        with pytest.raises(FluidSolverError) as e:
            call()
        assert e.value.status == FS_ERR_NAN
    col.position[5] = good[5]
    s.data.notify_that_data_changed()
    assert s.run(3).status == 0
    s.close()
