"""CM3D's half lists in grids of three and more cells per axis, where stencil cells wholly out of an atom's reach are
skipped: atoms on the cells' faces and edges, cells of unequal widths, a sheared grid (nothing skipped), with charges and
without.  The plain engine's four lists are the oracle's, pair for pair."""
import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from oracle import Oracle
from test_list_kernels import pair_keys

pytestmark = pytest.mark.gpu


def on_faces(natoms, shear, stretch, charged, shake):
    """FCC sites with one in the corner of the box, stretched along the axes, sheared, and moved by `shake` A"""
    wl = configs.lj_box(natoms, 0.8, 1.0, natoms, charged=charged)
    sysm = build_system(wl)
    m = np.diag(stretch)
    m[0, 1] = shear
    cells = int(np.ceil((sysm.natoms / 4) ** (1 / 3) - 1e-9))
    step = wl.box / (2 * cells)
    p = np.stack([sysm["px"], sysm["py"], sysm["pz"]]).astype(float)
    p = m @ (np.floor(p / step) * step)
    p += np.random.default_rng(natoms).normal(scale=shake, size=p.shape)
    sysm["px"], sysm["py"], sysm["pz"] = p
    sysm["hmat"] = (wl.box * m).ravel()
    return sysm


@pytest.mark.parametrize("natoms,shear,stretch,charged", [
    (864, 0.0, (1.0, 1.0, 1.0), False),
    (864, 0.0, (1.0, 1.0, 1.0), True),
    (2048, 0.0, (1.0, 1.3, 0.8), True),
    (4000, 0.0, (2.0, 1.0, 0.7), False),
    (4000, 0.15, (1.0, 1.0, 1.0), True),
])
@pytest.mark.parametrize("shake", [0.0, 0.2])
def test_half_lists(engine_lib, natoms, shear, stretch, charged, shake):
    sysm = on_faces(natoms, shear, stretch, charged, shake)
    n = sysm.natoms
    orc = Oracle(sysm.copy())
    orc.get_ngbr()
    with Engine(sysm.copy(), mode=_abi.PLAIN_FP64) as e:
        assert min(e.grid()[0]) >= 3
        e.get_ngbr()
        for w in range(4):
            np.testing.assert_array_equal(pair_keys(*e.pair_list(w), n), pair_keys(*orc.pair_list(w), n))
