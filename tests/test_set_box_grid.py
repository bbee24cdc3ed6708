"""A box that starts to move (cm3d_nb_set_box) takes the context back to CM3D's list radii: to their cell grid and, where
that grid has room for its windows, to the compact pair kernel, whichever grid the wider lists had.  Forces after the
change, with the lists carried over and with lists built anew, are the plain FP64 engine's in the new box to the mixed
engine's bound (1e-5 relative RMS; a mixed context made in the new box has another grid, hence other FP32 roundings);
replayed steps go on from there as that context's, to 1e-6 A after three of them (a step moves an atom by the forces'
share of some 0.05 A)."""
import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi
from cm3d_b200.engine import Engine
from test_list_grid import water
from test_list_kernels import slab

pytestmark = pytest.mark.gpu

# system, cells of the engine's own lists, cells of CM3D's, tuned before the box moves
CASES = {
    "water-8232": (lambda: water(14, 0.5), [3, 3, 3], [4, 4, 4], False),
    "water-8232, tuned": (lambda: water(14, 0.5), [3, 3, 3], [4, 4, 4], True),
    "water-17496": (lambda: water(18, 0.5), [4, 4, 4], [5, 5, 5], False),
    "water-12288, tuned": (lambda: water(16, 0.5), [4, 4, 4], [4, 4, 4], True),
    "slab 6 x 9 x 12": (lambda: slab(6, 9, 12), [3, 5, 6], [3, 5, 7], False),
}


@pytest.mark.parametrize("name", list(CASES))
def test_grid_and_kernel_go_back(engine_lib, name):
    make, wide, cells, tuned = CASES[name]
    sysm = make()
    h = np.asarray(sysm["hmat"], float)
    e = Engine(sysm, mode=_abi.MIXED)
    e.step_init()
    if tuned:
        e.autotune()
    assert e.grid()[0] == wide
    e.step(1, 3)
    pos, vel = e.positions(), e.velocities()
    f = 1.002
    e.set_box(f * h)
    assert e.grid()[0] == cells
    e.set_positions(f * pos)
    e.force(1)
    carried = e.forces(_abi.FXL)
    assert tuned or e.pair_kernel()[0] == "compact"
    e.step_init()
    built = e.forces(_abi.FXL)
    e.step(1, 3)
    after = e.positions()
    assert e.status()["nonfinite"] == 0 and e.status()["stage_timeouts"] == 0
    e.close()
    sysm["hmat"] = f * h
    sysm["px"], sysm["py"], sysm["pz"] = f * pos
    sysm["vx"], sysm["vy"], sysm["vz"] = vel
    with Engine(sysm, mode=_abi.MIXED) as e:
        e.step_init()
        e.step(1, 3)
        np.testing.assert_allclose(after, e.positions(), rtol=0, atol=1e-6)
    with Engine(sysm, mode=_abi.PLAIN_FP64) as e:
        e.step_init()
        exact = e.forces(_abi.FXL)
    assert rel_rms(built, exact) <= 1e-5
    assert rel_rms(carried, exact) <= 1e-5


def test_a_kernel_the_autotuner_left_stays_left(engine_lib, monkeypatch):
    """a context on another kernel by choice is not moved to the compact one"""
    sysm = water(16, 0.5)
    monkeypatch.setenv("CM3D_NB_PAIR_KERNEL", "window")
    e = Engine(sysm, mode=_abi.MIXED)
    e.get_ngbr()
    e.force(1)
    assert e.pair_kernel()[0] == "window"
    e.set_box(1.001 * np.asarray(sysm["hmat"], float))
    e.force(1)
    assert e.pair_kernel()[0] == "window"
    e.close()
