"""A step whose neighbor lists overflow the automatic capacity grows them and
starts over: the same state, bit for bit, as with lists that are large enough
from the start, the densities that the particles were uploaded with among it
(the first loop's viscosity reads them, and the boundary keeps them). And a
run that a NaN position ends leaves the densities as they were."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import scenes
from fluidsolver_b200._lib import FS_ERR_NAN, FluidSolverError
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu

IISPH = {2: [0.001, 2, 20, 0.5, 0.7, 0.01], 3: [0.001, 2, 20, 0.5, 0.7, 0.01, 1.0, 1.1]}


def dense_dam(dim, side):
    """A dam at a spacing that gives about 80 (3D) or 40 (2D) neighbors, with densities of its own."""
    if dim == 3:
        c, k = scenes.breaking_dam_3d(side, side, side, 1.0, tank=(2 * side, side + 4, side + 4), seed=side).collection, 0.75
    else:
        c, k = scenes.breaking_dam_2d(side, side, width=2 * side, height=side + 20, seed=side).collection, 0.55
    rng = np.random.default_rng(side)
    n = len(c)
    return ParticleCollection(position=np.ascontiguousarray(c.position * np.float32(k)),
                              velocity=rng.normal(0, 0.1, c.position.shape).astype(np.float32),
                              mass=np.full(n, k ** dim, np.float32),
                              density=rng.uniform(0.5, 1.5, n).astype(np.float32), type=c.type)


# the tile passes; eight threads per owner and one, stored gradients and none, in the device's order and the
# reference's; the small-scene kernel
CASES = [(3, 12, dict(precision="fp32-kahan")), (3, 12, dict(precision="fp32")),
         (3, 12, dict(precision="fp32", reference_order=True)), (3, 12, dict(precision="fp64")),
         (3, 41, dict(precision="fp32")), (3, 41, dict(precision="fp32", reference_order=True)),
         (2, 30, dict(precision="fp32-kahan")), (2, 30, dict(precision="fp32", reference_order=True)),
         (2, 190, dict(precision="fp32-kahan")), (2, 190, dict(precision="fp32", reference_order=True)),
         (2, 30, dict(precision="fp32-kahan", one_kernel_steps=True)),
         (2, 30, dict(precision="fp32", reference_order=True, one_kernel_steps=True))]


def solver(dim, **kw):
    return make_solver(f"iisph-{dim}d", "hashed-3d" if dim == 3 else "hashed-2d", IISPH[dim], (0.002, 0.4, 0.25), **kw)


@pytest.mark.parametrize("dim,side,kw", CASES)
def test_growing_the_lists_keeps_the_state(dim, side, kw):
    col = dense_dam(dim, side)
    res = []
    for capacity in (0, 128 if dim == 3 else 64):
        s = solver(dim, neighbor_capacity=capacity, **kw)
        s.data.collection = col
        st = s.step()
        assert st.max_neighbors > (64 if dim == 3 else 32)   # the automatic capacity overflows
        one = s.collection()
        st = s.run(3)
        res.append((st.iterations, one, s.collection()))
        s.close()
    (ia, *a), (ib, *b) = res
    assert ia == ib
    for x, y in zip(a, b):
        for f in ("position", "velocity", "acceleration", "density", "pressure"):
            assert bits_equal(getattr(x, f), getattr(y, f)), f
    boundary = col.type == 1
    assert bits_equal(a[0].density[boundary], col.density[boundary])


@pytest.mark.parametrize("dim,side,kw", CASES)
@pytest.mark.parametrize("steps", [1, 2, 4])
def test_a_run_that_an_error_ends_keeps_the_densities(dim, side, kw, steps):
    col = dense_dam(dim, side)
    col.position[17] = np.nan
    s = solver(dim, neighbor_capacity=128 if dim == 3 else 64, **kw)
    s.data.collection = col
    with pytest.raises(FluidSolverError) as e:
        s.run(steps)
    assert e.value.status == FS_ERR_NAN
    out = s.collection()
    for f in ("velocity", "mass", "density", "type"):
        assert bits_equal(getattr(out, f), getattr(col, f)), f
    s.close()
