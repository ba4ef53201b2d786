"""Compact hashing clamps cell coordinates to 31 bits: beyond them the three
cells of a row have one key, and the contract's walk lists that cell's members
once per cell. The exported lists hold each such neighbor as often, in
ascending order."""
import numpy as np
import pytest

from fluidsolver_b200 import NeighborhoodSearch
from fluidsolver_b200.solver import ParticleCollection

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,copies", [(3.0, 1), (1.5e9, 1), (3e9, 3), (-3e9, 3)])
@pytest.mark.parametrize("members", [2, 7, 13])
def test_members_of_clamped_cells(x, copies, members):
    pos = np.zeros((members + 3, 2), np.float32)
    pos[:members, 0] = x
    pos[members:, 0] = 17.0   # another cluster
    ns = NeighborhoodSearch("compact-hashing-2d", 2.0)
    ns.data.collection = ParticleCollection(position=pos)
    ns.find_neighbors()
    off, idx = ns.neighbor_lists()
    far, near = np.repeat(np.arange(members), copies), np.arange(members, members + 3)
    assert np.array_equal(np.diff(off), [len(far)] * members + [3] * 3)
    assert np.array_equal(idx, np.concatenate([far] * members + [near] * 3))
    ns.close()
