"""The search's order by counting against the radix sort's: the same stable
(region, cell) order, lists and cell walks. A scene takes the radix sort when
more than 1,024 excluded inactive particles lie in it, so the two paths run on
the same active particles with and without a crowd of inactive ones; further
sizes at the edges of the scan's tiles (4,096 entries), warps and blocks, and
dense cells on both sides of the line between the paths. And the lists built
with eight threads per owner against those with one (the small-scene kernel),
in place and order: the bit-exact state depends on both."""
import numpy as np
import pytest

from conftest import bits_equal
from fluidsolver_b200 import NeighborhoodSearch
from fluidsolver_b200.solver import ParticleCollection
from test_gpu_solvers import make_solver

pytestmark = pytest.mark.gpu
IIS3 = [0.001, 2, 8, 0.5, 0.7, 0.01, 1.0, 1.1]


def brute(pos, r, owners, candidates):
    out = []
    for i in range(len(pos)):
        if not owners[i]:
            out.append(np.empty(0, np.int64))
            continue
        d = (pos[i] - pos).astype(np.float32)
        q = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
        out.append(np.flatnonzero((q <= np.float32(r) * np.float32(r)) & candidates))
    return out


@pytest.mark.parametrize("n,spread,inactive", [(1, 3, 0), (2, 3, 1), (33, 4, 5), (257, 9, 0), (1000, 40, 1024),
                                               (1000, 40, 1025), (4000, 12, 0), (3000, 1.5, 0), (3000, 4.5, 7)])
def test_lists_on_both_paths(n, spread, inactive):
    rng = np.random.default_rng(n + inactive)
    pos = rng.uniform(-spread, spread, (n + inactive, 3)).astype(np.float32)
    typ = np.concatenate([rng.choice([0, 1], n), np.full(inactive, 2)]).astype(np.uint8)
    perm = rng.permutation(n + inactive)
    pos, typ = pos[perm], typ[perm]
    ns = NeighborhoodSearch("hashed-3d", 1.0)
    ns.data.collection = ParticleCollection(position=pos, type=typ)
    ns.find_neighbors()
    ns.find_neighbors()   # from the order of the first
    off, idx = ns.neighbor_lists()
    want = brute(pos, 1.0, typ != 2, typ != 2)
    assert np.array_equal(np.diff(off), [len(x) for x in want])
    assert np.array_equal(idx, np.concatenate(want))
    ns.close()


@pytest.mark.parametrize("precision,exact", [("fp32-kahan", False), ("fp32", True), ("fp64", False)])
def test_counting_and_radix_steps_are_the_same(precision, exact):
    rng = np.random.default_rng(3)
    g = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g + rng.uniform(-0.05, 0.05, g.shape)).astype(np.float32)
    n = len(pos)
    typ = (g[:, 1] == 0).astype(np.uint8)
    out = []
    for crowd in (0, 1500):   # inactive particles that no search lists; 1,500 take the radix sort
        p = np.concatenate([pos, rng.uniform(3, 9, (crowd, 3)).astype(np.float32)])
        s = make_solver("iisph-3d", "hashed-3d", IIS3, (0.005, 0.4, 0.25), precision=precision, reference_order=exact)
        s.data.collection = ParticleCollection(position=p, velocity=np.zeros_like(p), mass=np.ones(len(p), np.float32),
                                               density=np.ones(len(p), np.float32),
                                               type=np.concatenate([typ, np.full(crowd, 2, np.uint8)]))
        st = s.run(6)
        out.append((st.iterations, s.collection()))
        s.close()
    (ia, a), (ib, b) = out
    assert ia == ib
    for f in ("position", "velocity", "density", "pressure"):
        assert bits_equal(getattr(a, f)[:n], getattr(b, f)[:n]), f


@pytest.mark.parametrize("search,spacing", [("quadratic-2d", 1.0), ("quadratic-2d", 0.25), ("quadratic-2d", 0.11),
                                            ("hashed-2d", 0.25)])
def test_group_lists_keep_the_reference_order(search, spacing):
    """Lists of about 13, 200 and 1,000 entries: below, above and far above the 128 that are sorted together."""
    rng = np.random.default_rng(8)
    i, j = np.meshgrid(np.arange(40), np.arange(40), indexing="ij")
    pos = np.stack([i.ravel(), j.ravel()], 1) * spacing
    pos = (pos + rng.uniform(-0.03, 0.03, pos.shape)).astype(np.float32)[rng.permutation(1600)]
    out = []
    for one in (True, False):
        s = make_solver("sesph-2d", search, [1000.0, 0.01], (0.001, 0.4, 0.25), precision="fp32", reference_order=True,
                        one_kernel_steps=one, neighbor_capacity=1700)
        s.data.collection = ParticleCollection(position=pos.copy(), velocity=np.zeros_like(pos),
                                               mass=np.full(1600, spacing ** 2, np.float32),
                                               density=np.ones(1600, np.float32), type=np.zeros(1600, np.uint8))
        s.run(2)
        out.append(s.collection())
        s.close()
    for f in ("position", "velocity", "density", "pressure"):
        assert bits_equal(getattr(out[0], f), getattr(out[1], f)), f
