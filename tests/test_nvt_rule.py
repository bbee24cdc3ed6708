"""The thermostatted inner level on both sides of the rule between one cluster of blocks and grid-wide launches, for
molecules of several atoms: the last size in the cluster and the first beyond it, with one substep and with several,
and a few long molecules.  Plain FP64 engine against CM3D's algorithm (the oracle) after three steps, to the 1e-9 of the
other thermostat tests."""
import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from oracle import Oracle

pytestmark = pytest.mark.gpu


def chains(nmol, size, substeps):
    """argon atoms tied into chains of `size` by weak springs, under one Nose-Hoover chain"""
    n = nmol * size
    wl = configs.lj_box(n, 0.7, 1.0, n)
    sysm = build_system(wl)
    assert sysm.natoms == n
    i = np.arange(n, dtype=np.int32).reshape(nmol, size)
    sysm["ibond"], sysm["jbond"] = i[:, :-1].ravel().copy(), i[:, 1:].ravel().copy()
    sysm["nbonds"] = nmol * (size - 1)
    sysm["idxbond"], sysm["itypbond"] = np.zeros(nmol * (size - 1), np.int32), np.zeros(1, np.int32)
    sysm["eqbond"], sysm["fkbond"] = np.array([20.0]), np.array([1e-3])
    sysm["nres_intra"] = substeps
    gkt = np.array([3.0 * n * wl.temp, wl.temp, wl.temp])
    sysm["iensemble"], sysm["ntherm"], sysm["nchain"], sysm["ithm"] = 1, 1, 3, np.zeros(n, np.int32)
    sysm["gkt"], sysm["mnh"] = gkt, gkt * 0.08 ** 2
    sysm["nhc_eta"], sysm["nhc_veta"] = np.zeros(3), np.array([0.1, -0.2, 0.3])
    return sysm


@pytest.mark.parametrize("nmol,size,substeps", [(3072, 2, 1), (3074, 2, 1), (3413, 3, 4), (3414, 3, 4), (1024, 9, 1),
                                                (40, 64, 2)])
def test_molecules_on_both_sides(engine_lib, nmol, size, substeps):
    sysm = chains(nmol, size, substeps)
    with Engine(sysm.copy(), mode=_abi.PLAIN_FP64) as e:
        e.step_init()
        e.step(1, 3)
        eta, veta = e.nhc_state()
        pos = e.positions()
    o = Oracle(sysm.copy())
    o.step_init()
    o.step(1, 3)
    eo, vo = o.nhc_state()
    np.testing.assert_allclose(eta, np.asarray(eo).reshape(eta.shape), rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(veta, np.asarray(vo).reshape(eta.shape), rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(pos, o.positions(), rtol=0, atol=1e-9)
