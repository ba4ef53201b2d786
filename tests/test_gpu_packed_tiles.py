"""The pressure loop on packed tiles. A tile that fits the staging cap only without
padding between its ranges is staged packed, its pressures by plain stores to
memory that bulk copies fill next. How many tiles are packed follows the cap;
the separate passes, which stage once, take the same caps: the same sums in the
same order, so the state is the same bit for bit."""
import pytest

from conftest import bits_equal
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6000, 37889, 90000])
@pytest.mark.parametrize("cap", [1280, 1400, 1480, 1536])
def test_packed_tiles(n, cap):
    col = dam(n, n % 97)
    res = []
    for eager in (False, True):
        s = make_solver("iisph-3d", "hashed-3d", [0.001, 6, 6, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                        precision="fp32-kahan", sync_each_iteration=eager)
        s.data.collection = col
        s.initialize()
        s.set_tuning(1, 3, tile_cap=cap)
        s.step()
        s.step()
        res.append(s.collection())
        s.close()
    a, b = res
    for f in ("position", "velocity", "acceleration", "density", "pressure"):
        assert bits_equal(getattr(a, f), getattr(b, f)), f
