"""The thermostatted inner level in one cluster of blocks and as grid-wide launches: groups at the edges of the blocks
and of the rule between the two, one thermostat and as many as there are chunks to share out, each atom of a third
without one.  Plain FP64 engine against CM3D's algorithm (the oracle) after five steps, to the 1e-9 of the other
thermostat tests."""
import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from oracle import Oracle

pytestmark = pytest.mark.gpu


def chains(wl, ntherm):
    sysm = build_system(wl)
    n = sysm.natoms
    ithm = np.arange(n, dtype=np.int32) % (ntherm + 1 if ntherm > 1 else 1)
    ithm[ithm == ntherm] = -1
    gkt = np.tile([3.0 * n / ntherm * wl.temp, wl.temp, wl.temp], ntherm)
    sysm["iensemble"], sysm["ntherm"], sysm["nchain"], sysm["ithm"] = 1, ntherm, 3, ithm
    sysm["gkt"], sysm["mnh"] = gkt, gkt * 0.08 ** 2
    sysm["nhc_eta"], sysm["nhc_veta"] = np.zeros(3 * ntherm), np.tile([0.1, -0.2, 0.3], ntherm)
    return sysm


@pytest.mark.parametrize("natoms,ntherm", [(64, 1), (65, 2), (1025, 3), (4096, 1), (4096, 40), (4097, 2)])
def test_chains_at_the_edges(engine_lib, natoms, ntherm):
    sysm = chains(configs.lj_box(natoms, 0.7, 1.0, natoms), ntherm)
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
