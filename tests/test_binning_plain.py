"""The FP64 engine's binning on both sides of its rule (atoms times atoms per cell): the last water box of one cluster of
blocks, the first of the grid-wide kernels, and a box whose cells are many and small.  CM3D's lists are the oracle's,
pair for pair."""
import numpy as np
import pytest

from cm3d_b200 import _abi
from cm3d_b200.engine import Engine
from oracle import Oracle
from test_list_kernels import pair_keys, slab, water

pytestmark = pytest.mark.gpu

CASES = {
    "water-5184, 995,000": lambda: water(12),
    "water-6591, 1,609,000": lambda: water(13),
    "argon-12,000, 240,000": lambda: slab(10, 10, 30),
}


@pytest.mark.parametrize("name", list(CASES))
def test_lists_of_both_forms(engine_lib, name):
    sysm = CASES[name]()
    n = sysm.natoms
    orc = Oracle(sysm)
    orc.get_ngbr()
    with Engine(sysm, mode=_abi.PLAIN_FP64) as e:
        e.get_ngbr()
        lists = [e.pair_list(w) for w in range(4)]
    for w in range(4):
        np.testing.assert_array_equal(pair_keys(*lists[w], n), pair_keys(*orc.pair_list(w), n))
