"""The pressure iterations in one cooperative launch against the host-driven
loop of separate passes (FS_FLAG_SYNC_EACH_ITERATION): the same sums in the same
order, so the state is the same bit for bit, at the edges of its forms on a
148-SM device: one tile, a ragged last tile, the last size with a block per
tile (2 and 3 per SM), several tiles per block, and the graph's loop beyond
4,096 tiles. Iteration limits at their edges, and longer lists than usual."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import scenes
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


def dam(n, seed):
    """n fluid particles of a jittered block in its tank."""
    side = int(np.ceil(n ** (1 / 3)))
    sc = scenes.breaking_dam_3d(side, side, side, 1.0, tank=(2 * side, side + 4, side + 4), seed=seed)
    c = sc.collection
    keep = np.concatenate([np.arange(n), np.arange(sc.n_fluid, len(c))])
    return ParticleCollection(**{f: getattr(c, f)[keep] for f in ("position", "velocity", "mass", "density", "type")})


@pytest.mark.parametrize("n,min_it,max_it,capacity", [
    (100, 2, 100, 0), (129, 2, 100, 0), (5000, 2, 100, 0), (5000, 1, 1, 0), (5000, 2, 2, 0), (5000, 3, 3, 0),
    (5000, 7, 7, 256), (37888, 2, 9, 0), (37889, 2, 9, 0), (56832, 2, 9, 0), (56833, 2, 9, 0), (75777, 2, 9, 0),
    (524289, 2, 4, 0)])
def test_one_launch_equals_the_separate_passes(n, min_it, max_it, capacity):
    col = dam(n, n % 97)
    res = []
    for eager in (False, True):
        s = make_solver("iisph-3d", "hashed-3d", [0.001, min_it, max_it, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                        precision="fp32-kahan", sync_each_iteration=eager, neighbor_capacity=capacity)
        s.data.collection = col
        st = [(x.iterations, x.actual_dt, x.avg_density_error) for x in (s.step(), s.step())]
        res.append((st, s.collection()))
        s.close()
    (sa, a), (sb, b) = res
    for x, y in zip(sa, sb):
        assert x[0] == y[0] and bits_equal(np.float32(x[1]), np.float32(y[1]))
        assert x[2] == pytest.approx(y[2], rel=1e-6)   # a double sum in another order, rounded to float
    for f in ("position", "velocity", "acceleration", "density", "pressure"):
        assert bits_equal(getattr(a, f), getattr(b, f)), f
