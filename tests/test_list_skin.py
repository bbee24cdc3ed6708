"""The engine's own lists reach beyond CM3D's and are built less often: until an atom has moved half their skin
the pairs within the cut-offs must all be in them, while nrefsh's answer and CM3D's lists stay CM3D's.  A smooth
compression wave moves neighbours at cut-off distance by up to twice its amplitude against one another; the real-space
Ewald term is left strong at the cut-off, so that a missing pair shows.  The forces must be those of a context made at
the moved positions, to FP32 summation order (1e-6 relative RMS)."""
import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from test_list_kernels import binary, shaken, slab

pytestmark = pytest.mark.gpu

FXL = _abi.FXL


def water(ngrid, skin, frac=0.45):
    L = ngrid * configs.WATER_SPACING
    rc = min(10.0, frac * L)
    return build_system(shaken(configs.water_box(ngrid=ngrid, seed=ngrid, rc=rc, alpha=1.0 / rc, kmax=3, skin=skin,
                                                 placement="octant"), 1, 0.02))


CASES = {
    "water-648, two-radius box": lambda: water(6, 0.3),
    "water-1029, room for a skin": lambda: water(7, 0.3, 0.36),
    "water-3993 (3 cells)": lambda: water(11, 0.5),
    "water-5184, skin 1.5": lambda: water(12, 1.5),
    "water-12288": lambda: water(16, 0.5),
    "slab 5 x 6 x 9": lambda: slab(5, 6, 9),
    "binary-2047": lambda: binary(2047),
}


def wave(sysm, amplitude):
    """every atom moved along x by at most `amplitude`, a function of its place along x only"""
    pos = np.stack([sysm["px"], sysm["py"], sysm["pz"]]).astype(float)
    L = np.asarray(sysm["hmat"], float).reshape(3, 3)[0, 0]
    pos[0] += amplitude * np.sin(2.0 * np.pi * pos[0] / L)
    return pos


def moved_and_fresh(sysm, pos, istep):
    e = Engine(sysm, mode=_abi.MIXED)
    e.get_ngbr()
    e.set_positions(pos)
    rebuilt = e.nrefsh(istep)
    e.force(1)
    f = e.forces(FXL)
    e.get_ngbr()
    e.force(1)
    g = e.forces(FXL)
    n = e.status()["rebuilds"]
    e.close()
    return f, g, bool(rebuilt), n


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("part", [0.3, 0.98, 1.3])
def test_no_pair_is_missing_until_the_lists_are_built(engine_lib, name, part):
    sysm = CASES[name]()
    # half the skin of the engine's lists, if the box has room for it
    half = 0.5 * max(0.2 * float(np.sqrt(np.max(sysm["rmaxl_cut2"]))), float(sysm["skin"]))
    pos = wave(sysm, part * half)
    f, g, rebuilt, builds = moved_and_fresh(sysm, pos, 100)
    d = np.max(np.abs(pos[0] - sysm["px"]))
    assert rebuilt == (d > 0.5 * float(sysm["skin"]))
    assert builds == 2 + int(rebuilt)
    assert rel_rms(f, g) <= 1e-6


@pytest.mark.parametrize("shrink", [0.99, 0.94])
def test_a_box_that_moves_goes_back_to_the_thin_skin(engine_lib, shrink):
    sysm = water(12, 0.5)
    h = np.asarray(sysm["hmat"], float)
    pos = shrink * np.stack([sysm["px"], sysm["py"], sysm["pz"]]).astype(float)
    e = Engine(sysm, mode=_abi.MIXED)
    e.get_ngbr()
    e.force(1)
    e.set_box(shrink * h)
    e.set_positions(pos)
    assert e.nrefsh(100)
    e.force(1)
    f = e.forces(FXL)
    e.close()
    sysm["hmat"] = shrink * h
    sysm["px"], sysm["py"], sysm["pz"] = pos
    e = Engine(sysm, mode=_abi.MIXED)
    e.get_ngbr()
    e.force(1)
    assert rel_rms(f, e.forces(FXL)) <= 1e-6
    e.close()


def test_staged_lists_of_a_large_batch(engine_lib, monkeypatch):
    """152,000 atoms: the staged list kernel's side of its rule, bit for bit the warp-per-atom walk"""
    sysm = [binary(2047), build_system(shaken(configs.lj_box(4096, 0.8, 1.0, 7), 7))] * 25
    out = []
    for walk in (False, True):
        if walk:
            monkeypatch.setenv("CM3D_NB_LIST_KERNEL", "walk")
        e = Engine(sysm, mode=_abi.MIXED)
        e.get_ngbr()
        e.force(1)
        out.append(e.forces(FXL))
        assert e.status()["nonfinite"] == 0
        e.close()
    np.testing.assert_array_equal(out[0], out[1])
