"""A batch's systems in coarse grids (fewer than 3 cells along an axis) on both sides of the size from which their list
skin is the thin one, among systems of finer grids: forces after steps that rebuild at each system's own time are the
plain FP64 engine's at the same positions, to the mixed engine's bound (1e-5 relative RMS)."""
import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system

pytestmark = pytest.mark.gpu


def water(ngrid, skin=0.5):
    return build_system(configs.water_box(ngrid=ngrid, seed=ngrid, rc=10.0, alpha=0.31, kmax=5, skin=skin,
                                          placement="octant"))


def lj(natoms, skin_of_cut, charged):
    sysm = build_system(configs.lj_box(natoms, 0.8, 1.5, natoms, charged=charged))
    cut = float(np.sqrt(np.max(sysm["rmaxl_cut2"])))
    sysm["skin"] = skin_of_cut * cut
    for k in ("rmaxs", "rmaxl"):
        sysm[k + "_skin2"] = (np.sqrt(np.asarray(sysm[k + "_cut2"])) + sysm["skin"]) ** 2
    if charged:
        for k, c in (("rmaxs_skin2_e", "rmaxs_coul2"), ("rmaxl_skin2_e", "rmaxl_coul2")):
            sysm[k] = (np.sqrt(sysm[c]) + sysm["skin"]) ** 2
    return sysm


CASES = {
    "water 375, 648, 1536": lambda: [water(5), water(6), water(8)],
    "water 1029": lambda: [water(7), water(7, 1.0), water(6)],
    "water 1536 at 0.5, 1 and 1.5 A, and 3993": lambda: [water(8), water(8, 1.0), water(8, 1.5), water(11)],
    "charged 510, 512, 514": lambda: [lj(n, 0.06, True) for n in (510, 512, 514)],
    "argon 512, 513, 2048": lambda: [lj(n, 0.06, False) for n in (512, 513, 2048)],
}


@pytest.mark.parametrize("name", list(CASES))
def test_forces_after_steps(engine_lib, name):
    systems = CASES[name]()
    with Engine([s.copy() for s in systems], mode=_abi.MIXED) as e:
        e.step_init()
        e.step(1, 40)
        pos, f = e.positions(), e.forces(_abi.FXL)
        ranges = list(e.ranges)
        assert min(e.system_counts()[0]) > 1                  # every system's schedule has rebuilt
        assert e.status()["nonfinite"] == 0
    for s, (a, n) in zip(systems, ranges):
        with Engine(s.copy(), mode=_abi.PLAIN_FP64) as p:
            p.set_positions(pos[:, a:a + n])
            p.step_init()
            assert rel_rms(f[:, a:a + n], p.forces(_abi.FXL)) <= 1e-5
