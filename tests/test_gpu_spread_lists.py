"""The order of the tile lists' entries: spread over the shared-memory banks, or,
when the lists are too long for the memory that the sorting needs (a capacity
of 256 here) or on a 148-SM device up to 75,776 owners, as the rows of cells
give them. The lists hold the same entries,
so the results differ by the rounding of the sums alone: a density is a
compensated sum of partial sums of 8 terms (8 roundings of 2^-24 on either
side, 1e-6); a velocity hangs on the density's difference from the rest
density, at least a hundredth of it (1e-4)."""
import numpy as np
import pytest

from fluidsolver_b200.solver import ParticleCollection
from test_gpu_pressure_loop import dam
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spacing,capacity", [
    (75776, 1.0, 0), (75777, 1.0, 0), (80001, 1.0, 104), (80001, 0.85, 88), (80001, 0.8, 120)])
def test_spread_lists_hold_the_same_entries(n, spacing, capacity):
    col = dam(n, n % 89)
    col.position = np.ascontiguousarray(col.position * np.float32(spacing))
    res = []
    for cap in (capacity, 256):
        s = make_solver("iisph-3d", "hashed-3d", [0.001, 1, 1, 0.5, 0.7, 0.01, 1.0, 1.1], (0.005, 0.4, 0.25),
                        precision="fp32-kahan", neighbor_capacity=cap)
        s.data.collection = ParticleCollection(**{f: getattr(col, f) for f in
                                                  ("position", "velocity", "mass", "density", "type")})
        s.step()
        res.append(s.collection())
        s.close()
    a, b = res
    fluid = col.type == 0   # the particles that have lists
    np.testing.assert_allclose(a.density[fluid], b.density[fluid], rtol=1e-6)
    np.testing.assert_allclose(a.velocity, b.velocity, rtol=0, atol=1e-4 * np.abs(b.velocity).max())
