"""The gather phases with eight threads per owner against those with one (the
small-scene kernel runs the one-thread functions): the same state bit for bit,
at list lengths on both sides of the 32 entries that are in flight together
and of twice as many, with list lengths from one upwards in the same warps,
boundary neighbors, and inactive particles among the owners' warps."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import _lib as F
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu

SETTINGS = {"sesph-2d": [1000.0, 0.01], "iisph-2d": [0.001, 2, 100, 0.5, 0.7, 0.01],
            "sesph-3d": [1000.0, 0.01, 1, 1.1, 1.1], "iisph-3d": [0.001, 2, 20, 0.5, 0.7, 0.01, 1.0, 1.1]}


@pytest.mark.parametrize("precision,exact", [("fp32", True), ("fp64", False), ("fp32-kahan", False), ("fp32", False)])
@pytest.mark.parametrize("solver,search", [("sesph-2d", "hashed-2d"), ("iisph-2d", "quadratic-2d"),
                                           ("sesph-3d", "hashed-3d"), ("iisph-3d", "quadratic-3d")])
@pytest.mark.parametrize("spacing", [1.0, 0.75])
def test_groups_equal_single_threads(solver, search, precision, exact, spacing):
    if solver.endswith("3d") and precision == "fp32-kahan":
        pytest.skip("the 3D fast mode runs on tile lists")
    rng = np.random.default_rng(17)
    dim = 2 if solver.endswith("2d") else 3
    m = 20 if dim == 2 else 8
    block = np.stack(np.meshgrid(*[np.arange(m)] * dim, indexing="ij"), -1).reshape(-1, dim) * spacing
    pos = np.concatenate([block + rng.uniform(-0.05, 0.05, block.shape),
                          rng.uniform(-4, m + 4, (150, dim))]).astype(np.float32)   # stragglers: short lists
    n = len(pos)
    typ = rng.choice([0, 0, 0, 0, 1, 2] if solver != "iisph-2d" else [0, 0, 0, 1], n).astype(np.uint8)
    vel = rng.normal(0, 0.3, (n, dim)).astype(np.float32) * (typ == 0)[:, None]
    col = dict(position=pos, velocity=vel.astype(np.float32), mass=np.full(n, spacing ** dim, np.float32),
               density=np.ones(n, np.float32), type=typ)
    out = []
    for one in (True, False):
        s = make_solver(solver, search, SETTINGS[solver], (0.001, 0.4, 0.25), precision=precision, reference_order=exact,
                        one_kernel_steps=one, neighbor_capacity=160)
        s.data.collection = ParticleCollection(**{k: v.copy() for k, v in col.items()})
        st = s.run(4)
        assert (F.lib().fs_small_blocks(s.ctx) > 0) == one
        out.append((st.iterations, np.float32(st.actual_dt), s.collection(), st.max_neighbors))
        s.close()
    (ia, da, a, ma), (ib, db, b, mb) = out
    assert ia == ib and bits_equal(da, db) and ma == mb
    if spacing < 1 and dim == 3:
        assert ma > 64
    for f in ("position", "velocity", "acceleration", "density", "pressure"):
        assert bits_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("precision,exact", [("fp32", True), ("fp64", False), ("fp32", False)])
def test_stored_gradients_keep_the_sums(precision, exact):
    """Both forms of the pressure passes on stored gradients (eight threads per owner up to 20,480 fluid particles, one
    beyond) and both forms of the first loop that stores them (up to 65,536, in FP64 45,056) against each other: the
    same block of fluid alone and with as many far-away single particles as it takes to change the form."""
    rng = np.random.default_rng(23)
    m = 10
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    block = (g * 0.9 + rng.uniform(-0.03, 0.03, g.shape)).astype(np.float32)
    typ = (g[:, 1] == 0).astype(np.uint8)
    out = []
    for far in (0, 21000, 66000):
        side = int(np.ceil(far ** (1 / 3))) or 1
        grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:far]
        pos = np.concatenate([block, (grid * 5.0 + 30.0).astype(np.float32)])
        s = make_solver("iisph-3d", "hashed-3d", [0.001, 5, 5, 0.5, 0.7, 0.01, 1.0, 1.1], (0.001, 0.4, 0.25),
                        precision=precision, reference_order=exact)
        s.data.collection = ParticleCollection(position=pos, velocity=np.zeros_like(pos),
                                               mass=np.ones(len(pos), np.float32),
                                               density=np.ones(len(pos), np.float32),
                                               type=np.concatenate([typ, np.zeros(far, np.uint8)]))
        st = s.run(3)
        assert st.iterations == 5
        out.append(s.collection())
        s.close()
    n = len(block)
    for other in out[1:]:
        for f in ("position", "velocity", "acceleration", "density", "pressure"):
            assert bits_equal(getattr(out[0], f)[:n], getattr(other, f)[:n]), f
