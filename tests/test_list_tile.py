"""The tiled list kernel in the shapes that larger systems give it: 32 atoms to a block, more atom types than its table
of radii holds and more than a warp's lanes, cells fuller than the mean by more than its blocks' share.  CM3D's lists
are the oracle's, pair for pair; the full lists, seen through the forces, are bit for bit the warp-per-atom walk's.  The
tiled kernel writes the compact list itself, one launch fewer than the walk and its conversion."""
import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from oracle import Oracle
from test_halted_steps import stretched
from test_list_kernels import pair_keys, water

pytestmark = pytest.mark.gpu


def more_types(sysm, ntypes):
    """the same system with its two atom types split into `ntypes`"""
    old, n_old = np.asarray(sysm["itype"]), int(sysm["ntypes"])
    kind = np.arange(ntypes) % n_old                       # the old type of each new one
    itype = old.copy()
    for t in range(n_old):
        mine = np.flatnonzero(kind == t)
        at = np.flatnonzero(old == t)
        itype[at] = mine[np.arange(len(at)) % len(mine)]
    sysm["map"] = np.asarray(sysm["map"]).reshape(n_old, n_old)[np.ix_(kind, kind)].astype(np.int32).ravel()
    sysm["itype"], sysm["ntypes"] = itype.astype(np.int32), ntypes
    return sysm


def uneven():
    sysm, dense = stretched(configs.water_box(ngrid=16, seed=2, kmax=3, placement="octant"), 3, 2)
    sysm["px"], sysm["py"], sysm["pz"] = dense
    return sysm


CASES = {
    # the system, whether its compact list is written directly
    "water-12288, 32 atoms to a block": (lambda: water(16), True),
    "water-12288, 9 types": (lambda: more_types(water(16), 9), True),
    "water-5184, 33 types": (lambda: more_types(water(12), 33), False),
    "water-12288, 40 types": (lambda: more_types(water(16), 40), False),
    "half-filled box, cells of twice the mean": (uneven, True),
}


@pytest.mark.parametrize("name", list(CASES))
def test_tiles_against_the_walk_and_the_oracle(engine_lib, name, monkeypatch):
    make, direct = CASES[name]
    sysm = make()
    n = sysm.natoms
    out, launches = [], []
    for walk in (False, True):
        if walk:
            monkeypatch.setenv("CM3D_NB_LIST_KERNEL", "walk")
        with Engine(sysm, mode=_abi.MIXED) as e:
            e.get_ngbr()                                   # widens the slots where it has to
            before = e.launch_count()
            e.get_ngbr()
            launches.append(e.launch_count() - before)
            e.force(1)
            out.append(e.forces(_abi.FXL))
            assert e.status()["nonfinite"] == 0
            lists = [e.pair_list(w) for w in range(4)]
    assert launches[1] - launches[0] == int(direct)
    np.testing.assert_array_equal(out[0], out[1])
    orc = Oracle(sysm)
    orc.get_ngbr()
    for w in range(4):
        np.testing.assert_array_equal(pair_keys(*lists[w], n), pair_keys(*orc.pair_list(w), n))
