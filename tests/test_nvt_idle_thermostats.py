"""More thermostats than the first block of the cluster kernel has threads, most of them without an atom: the chains
that have atoms are turned by other blocks than the one that formed their kinetic sums, across a barrier of the whole
cluster.  Plain FP64 engine against CM3D's algorithm (the oracle), to the 1e-9 of the other thermostat tests."""
import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from oracle import Oracle

pytestmark = pytest.mark.gpu


def chains(natoms, ntherm, busy):
    """`natoms` argon atoms, dealt out among the thermostats `busy` of `ntherm`"""
    wl = configs.lj_box(natoms, 0.7, 1.0, natoms)
    sysm = build_system(wl)
    gkt = np.tile([3.0 * natoms / len(busy) * wl.temp, wl.temp, wl.temp], ntherm)
    sysm["iensemble"], sysm["ntherm"], sysm["nchain"] = 1, ntherm, 3
    sysm["ithm"] = np.asarray(busy, np.int32)[np.arange(natoms) % len(busy)]
    sysm["gkt"], sysm["mnh"] = gkt, gkt * 0.08 ** 2
    sysm["nhc_eta"], sysm["nhc_veta"] = np.zeros(3 * ntherm), np.tile([0.1, -0.2, 0.3], ntherm)
    return sysm


@pytest.mark.parametrize("natoms,ntherm,busy", [(128, 65, [64]), (128, 64, [63]), (1025, 600, [0, 400, 599]),
                                                (4096, 513, [512]), (64, 200, [199])])
def test_chains_of_other_blocks(engine_lib, natoms, ntherm, busy):
    sysm = chains(natoms, ntherm, busy)
    e = Engine(sysm.copy(), mode=_abi.PLAIN_FP64)
    e.step_init()
    e.step(1, 5)
    eta, veta = e.nhc_state()
    pos = e.positions()
    e.close()
    o = Oracle(sysm.copy())
    o.step_init()
    o.step(1, 5)
    eo, vo = o.nhc_state()
    np.testing.assert_allclose(eta, np.asarray(eo).reshape(eta.shape), rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(veta, np.asarray(vo).reshape(eta.shape), rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(pos, o.positions(), rtol=0, atol=1e-9)
