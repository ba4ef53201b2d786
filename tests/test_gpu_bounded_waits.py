"""The waits between the blocks of one launch, made to run out
(fs_set_grid_wait_limits): the search's scan, whose tiles wait for the tiles
before them, and the grid barriers of the pressure loop. A search that gives
up leaves the state as it was, bit for bit, and the context goes on as one that
never failed."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import _lib as F
from fluidsolver_b200 import scenes
from fluidsolver_b200._lib import FS_ERR_TIMEOUT, FluidSolverError
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu

IISPH3 = [0.001, 2, 9, 0.5, 0.7, 0.01, 1.0, 1.1]
MODES = {"tiles": ("iisph-3d", "hashed-3d", IISPH3, dict(precision="fp32-kahan")),
         "exact": ("iisph-3d", "hashed-3d", IISPH3, dict(precision="fp32", reference_order=True)),
         "fp64": ("iisph-3d", "hashed-3d", IISPH3, dict(precision="fp64")),
         "sesph": ("sesph-3d", "hashed-3d", [1000.0, 0.01, 1, 1.1, 1.1], dict(precision="fp32-kahan")),
         "2d": ("iisph-2d", "hashed-2d", IISPH3[:6], dict(precision="fp32-kahan")),
         "2d-history": ("iisph-2d", "hashed-2d", IISPH3[:6], dict(precision="fp32", reference_order=True))}
FIELDS = ("position", "velocity", "acceleration", "external", "mass", "density", "pressure", "type")


def solver(mode):
    name, search, settings, kw = MODES[mode]
    if name.endswith("2d"):
        col = scenes.breaking_dam_2d(60, 60, width=220, height=180, seed=3).collection
    else:
        col = dam(6000, 5)
    n = len(col)
    rng = np.random.default_rng(6)
    col = ParticleCollection(position=col.position, velocity=rng.normal(0, 0.1, col.position.shape).astype(np.float32),
                             mass=col.mass, density=rng.uniform(0.9, 1.1, n).astype(np.float32),
                             pressure=rng.uniform(0, 1, n).astype(np.float32), type=col.type)
    s = make_solver(name, search, settings, (0.001, 0.4, 0.25), **kw)
    s.data.collection = col
    return s


def limits(s, scan, barrier):
    F.check(F.lib().fs_set_grid_wait_limits(s.ctx, scan, barrier))


def fails(call):
    with pytest.raises(FluidSolverError) as e:
        call()
    assert e.value.status == FS_ERR_TIMEOUT


def same(a, b):
    for f in FIELDS:
        assert bits_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("mode", list(MODES))
def test_a_scan_that_gives_up_leaves_the_state(mode):
    s, other = solver(mode), solver(mode)
    limits(s, 0, -1)
    before = s.collection()
    for call in (s.step, s.execute_neighborhood_search, lambda: s.run(5), s.step):
        fails(call)
        same(s.collection(), before)
    limits(s, -1, -1)
    a, b = s.run(4), other.run(4)
    assert (a.iterations, a.actual_dt) == (b.iterations, b.actual_dt)
    same(s.collection(), other.collection())
    s.close()
    other.close()


def test_an_earlier_error_does_not_hide_it():
    """A position that is NaN is found before the scan; the table is incomplete all the same."""
    s = solver("tiles")
    s.data.collection.position[77] = np.nan
    limits(s, 0, -1)
    before = s.collection()
    for _ in range(2):
        fails(s.step)
        same(s.collection(), before)
    s.close()


def test_after_it_position_queries_need_a_search():
    s = solver("tiles")
    s.execute_neighborhood_search()
    assert len(s.get_neighbors_of_position([3.0, 3.0, 3.0])) > 0
    limits(s, 0, -1)
    fails(s.execute_neighborhood_search)
    with pytest.raises(FluidSolverError) as e:
        s.get_neighbors_of_position([3.0, 3.0, 3.0])
    assert e.value.status == F.FS_ERR_STATE
    limits(s, -1, -1)
    s.execute_neighborhood_search()
    assert len(s.get_neighbors_of_position([3.0, 3.0, 3.0])) > 0
    s.close()


@pytest.mark.parametrize("n", [6000, 90000])   # a block per tile, and several tiles per block
def test_a_barrier_that_gives_up_ends_the_step(n):
    s = make_solver("iisph-3d", "hashed-3d", IISPH3, (0.005, 0.4, 0.25), precision="fp32-kahan")
    s.data.collection = dam(n, 5)
    s.step()
    before = s.collection()
    limits(s, -1, 0)
    fails(s.step)
    mid = s.collection()   # the step ended before its integration
    for f in ("position", "velocity", "mass", "type"):
        assert bits_equal(getattr(mid, f), getattr(before, f)), f
    limits(s, -1, -1)
    st = s.step()
    assert st.status == 0 and 2 <= st.iterations <= 9
    assert np.isfinite(s.collection().position).all()
    s.close()
