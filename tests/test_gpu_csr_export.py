"""fs_get_neighbors_csr at the edges of its sorting kernels: list lengths around
a warp's 32 lanes, the longest list a warp ranks (512), the longest list
sorted in shared memory (8,192) and past it. Clusters of particles, every
member within the radius of every other and of no other cluster's, so each
owner's list is exactly its cluster, ascending."""
import numpy as np
import pytest

from fluidsolver_b200 import NeighborhoodSearch
from fluidsolver_b200.solver import ParticleCollection

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,owners", [((1, 2, 31, 32, 33, 64, 65), 3), ((511, 512, 513, 7), 3),
                                          ((8191, 8192, 8193, 40), 3), ((4200, 5, 600), 4200)])
def test_lists_are_the_sorted_clusters(sizes, owners):
    rng = np.random.default_rng(sum(sizes))
    cluster = np.repeat(np.arange(len(sizes)), sizes)
    n = len(cluster)
    # hashed-2d: fluid owners, every particle a candidate; 4,200 owners of a cluster are 17.6 million entries,
    # more than one chunk of the export
    first = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    fluid = np.arange(n) - first[cluster] < owners
    pos = np.stack([cluster * 10.0, np.zeros(n)], 1) + rng.uniform(-0.3, 0.3, (n, 2))
    perm = rng.permutation(n)
    pos, cluster, fluid = pos[perm].astype(np.float32), cluster[perm], fluid[perm]
    ns = NeighborhoodSearch("hashed-2d", 1.0)
    ns.data.collection = ParticleCollection(position=pos, type=np.where(fluid, 0, 1).astype(np.uint8))
    ns.find_neighbors()
    for _ in range(2):   # the second call reuses the kept workspace
        off, idx = ns.neighbor_lists()
        want = [np.flatnonzero(cluster == cluster[i]) if fluid[i] else np.empty(0, np.int64) for i in range(n)]
        assert np.array_equal(np.diff(off), [len(x) for x in want])
        assert np.array_equal(idx, np.concatenate(want))
    ns.close()
