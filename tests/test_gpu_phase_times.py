"""The phase times of a step, which its kernels note themselves in the graph
paths (a whole step, several steps, search and step by themselves) and events
measure in the host-driven one: not negative, positive for the phases that the
solver has, and together no longer than the calls took."""
import time

import numpy as np
import pytest

from fluidsolver_b200 import _lib as F, scenes
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu

IISPH = [0.001, 2, 100, 0.5, 0.7, 0.01, 1.0, 1.1]
SESPH = [1000.0, 0.01, 1.0, 1.1, 1.1]


@pytest.mark.parametrize("kind,search,settings,precision,phases", [
    ("iisph-3d", "hashed-3d", IISPH, "fp32-kahan", (0, 1, 2, 3, 4)),
    ("iisph-3d", "compressed-3d", IISPH, "fp64", (0, 1, 2, 3, 4)),
    ("iisph-2d", "hashed-2d", IISPH, "fp32", (0, 1, 2, 3, 4)),
    ("sesph-2d", "hashed-2d", SESPH, "fp32-kahan", (0, 1, 2, 4)),
    ("sesph-3d", "hashed-3d", SESPH, "fp32-kahan", (0, 1, 2, 3, 4))])
@pytest.mark.parametrize("eager", [False, True])
def test_phase_times(kind, search, settings, precision, phases, eager):
    col = dam(3000, 5) if "3d" in kind else scenes.breaking_dam_2d(40, 40, width=100, height=60).collection
    s = make_solver(kind, search, settings, (0.005, 0.4, 0.25), precision=precision, sync_each_iteration=eager)
    s.data.collection = col
    s.step()

    def search_and_step():
        F.check(F.lib().fs_find_neighbors(s.ctx))
        F.check(F.lib().fs_solve_step(s.ctx, 0.005, None))

    for call in (s.step, lambda: s.run(3), search_and_step):
        t = time.perf_counter()
        call()
        wall = (time.perf_counter() - t) * 1e3
        ms = np.asarray(s.phase_times())
        assert (ms >= 0).all() and all(ms[i] > 0 for i in phases) and ms.sum() <= wall, (ms, wall)
    s.close()
