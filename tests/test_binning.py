"""Binning by one cluster of blocks per system and by the grid-wide kernels: systems at the edges of the blocks'
threads (an atom, a thread), of the clusters and of the rule between the two, cells of a few atoms up to one cell that
holds the whole box.  CM3D's lists must be the oracle's, pair for pair, and the forces repeat bit for bit (the order of
a cell's atoms does not depend on the order of arrival)."""
import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from oracle import Oracle
from test_list_kernels import pair_keys, shaken, slab

pytestmark = pytest.mark.gpu


def box(n):
    return build_system(shaken(configs.lj_box(n, 0.7, 1.0, n), n))


CASES = {
    "3 atoms, one cell": lambda: box(3),
    "108": lambda: box(108),
    "1023": lambda: box(1023),
    "1024": lambda: box(1024),
    "1025": lambda: box(1025),
    "8193": lambda: box(8193),
    "32768, 4 atoms per thread": lambda: slab(16, 16, 32),
    "33792, grid-wide kernels": lambda: slab(16, 16, 33),
}


@pytest.mark.parametrize("name", list(CASES))
def test_cells_at_the_edges(engine_lib, name):
    sysm = CASES[name]()
    n = sysm.natoms
    orc = Oracle(sysm)
    orc.get_ngbr()
    runs = []
    for _ in range(2):
        e = Engine(sysm, mode=_abi.MIXED)
        e.get_ngbr()
        e.force(1)
        runs.append(e.forces(_abi.FXL))
        lists = [e.pair_list(w) for w in range(2)]
        e.close()
    np.testing.assert_array_equal(*runs)
    for w in range(2):
        np.testing.assert_array_equal(pair_keys(*lists[w], n), pair_keys(*orc.pair_list(w), n))
