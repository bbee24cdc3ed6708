"""Small sheared boxes whose atoms sit on lattice sites: many pairs lie exactly half a box apart along a box vector,
where FP32 cannot tell which of two images CM3D takes, and in a sheared box the two are not equally long.  CM3D's lists
must be the oracle's, pair for pair, in both engines, and level-1 forces its forces (plain 1e-11, mixed 1e-5 relative
RMS).  With a shear of 0.6 such pairs lie within the cut-off; there the mixed pair kernels, which follow a near pair's
image in FP32, take one image or the other, and only the plain engine's forces are held."""
import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from oracle import Oracle
from test_list_kernels import pair_keys

pytestmark = pytest.mark.gpu


def sheared(natoms, density, shear, skin, stretch=(1.0, 1.0, 1.0), charged=False):
    """FCC sites, some empty, in a box sheared by `shear` = (xy, xz, yz) and stretched along its edges, with lists of
    `skin` beyond the cut-offs"""
    wl = configs.lj_box(natoms, density, 1.0, natoms, charged=charged)
    sysm = build_system(wl)
    m = np.eye(3)
    m[0, 1], m[0, 2], m[1, 2] = shear
    m = m @ np.diag(stretch)
    cells = int(np.ceil((sysm.natoms / 4) ** (1 / 3) - 1e-9))
    step = wl.box / (2 * cells)                              # half an FCC cell
    p = np.stack([sysm["px"], sysm["py"], sysm["pz"]]).astype(float)
    sysm["px"], sysm["py"], sysm["pz"] = m @ ((np.floor(p / step) + 0.5) * step)
    sysm["hmat"] = (wl.box * m).ravel()
    sysm["skin"] = skin
    for k in ("rmaxs", "rmaxl"):
        sysm[k + "_skin2"] = (np.sqrt(np.asarray(sysm[k + "_cut2"])) + skin) ** 2
    if charged:
        for k, cut in (("rmaxs_skin2_e", "rmaxs_coul2"), ("rmaxl_skin2_e", "rmaxl_coul2")):
            sysm[k] = (np.sqrt(sysm[cut]) + skin) ** 2
    return sysm


CASES = {
    "60": lambda: sheared(60, 0.5, (-0.04, 0.03, -0.09), 2.5),
    "92, charged": lambda: sheared(92, 0.5, (-0.14, 0.04, 0.08), 2.5, charged=True),
    "68, charged, skin 1": lambda: sheared(68, 0.5, (0.16, 0.15, -0.05), 1.0, charged=True),
    "60, shear 0.6": lambda: sheared(60, 0.36, (0.6, 0.0, 0.0), 1.0),
    "60, shear 0.6 and -0.5, charged": lambda: sheared(60, 0.36, (0.6, 0.0, -0.5), 1.0, charged=True),
    "200, long along z": lambda: sheared(200, 0.6, (0.2, -0.1, 0.1), 4.0, (1.0, 1.0, 3.0)),
    "200, long along x": lambda: sheared(200, 0.6, (0.5, 0.1, -0.3), 4.0, (2.5, 1.0, 1.0)),
    "60, cubic": lambda: sheared(60, 0.5, (0.0, 0.0, 0.0), 2.5),
}


@pytest.mark.parametrize("name", list(CASES))
def test_pairs_half_a_box_apart(engine_lib, name):
    sysm = CASES[name]()
    n = sysm.natoms
    orc = Oracle(sysm.copy())
    orc.step_init()
    want = [pair_keys(*orc.pair_list(w), n) for w in range(4)]
    ref = orc.forces(0)
    # the forces of a lattice are small differences; those of the atoms moved by 0.1 A set the scale
    moved = sysm.copy()
    for k, d in zip(("px", "py", "pz"), np.random.default_rng(1).normal(scale=0.1, size=(3, n))):
        moved[k] = np.asarray(sysm[k]) + d
    shaken = Oracle(moved)
    shaken.step_init()
    scale = float(np.sqrt((shaken.forces(0) ** 2).mean()))
    for mode, tol in ((_abi.PLAIN_FP64, 1e-11), (_abi.MIXED, 1e-5)):
        with Engine(sysm.copy(), mode=mode) as e:
            e.step_init()
            f = e.forces(_abi.FXL)
            for w in range(4):
                np.testing.assert_array_equal(pair_keys(*e.pair_list(w), n), want[w])
        if mode == _abi.PLAIN_FP64 or "shear 0.6" not in name:
            assert rel_rms(f, ref, scale) <= tol
