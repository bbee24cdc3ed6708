"""The list kernels over the grids where their FP32 tests could go wrong: boxes of one, two and three or more
cells per axis (minimum image in the test, near-image pairs), axes of different cell counts, cells of a few and
of hundreds of atoms (the staged, the tiled and the warp-per-atom kernel), molecules with exclusions, several
types.  CM3D's half lists must be the oracle's, pair for pair; the full lists are seen through the forces: bit for
bit those of the warp-per-atom walk, which shares the decisions but neither the staging nor the order of work, and
within the mixed engine's bound (1e-5 relative RMS) of the plain FP64 engine's."""
import dataclasses

import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from oracle import Oracle

pytestmark = pytest.mark.gpu


def shaken(wl, seed, scale=0.15):
    rng = np.random.default_rng(seed)
    return dataclasses.replace(wl, pos=wl.pos + np.clip(rng.normal(scale=scale, size=wl.pos.shape), -0.4, 0.4))


def water(ngrid, skin=0.5):
    L = ngrid * configs.WATER_SPACING
    rc = min(10.0, 0.45 * L)
    return build_system(shaken(configs.water_box(ngrid=ngrid, seed=ngrid, rc=rc, alpha=3.1 / rc, kmax=3, skin=skin,
                                                 placement="octant"), 1, 0.02))


def slab(nx, ny, nz, seed=3):
    """argon in an orthorhombic box of nx x ny x nz FCC cells: axes of different cell counts"""
    a = (4.0 / 0.8442) ** (1.0 / 3.0) * configs.ARGON["sig"]
    wl = configs.argon_fcc(ncell=1, seed=seed)
    cells = np.array([(i, j, k) for i in range(nx) for j in range(ny) for k in range(nz)], dtype=float)
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]]) + 0.25
    pos = ((cells[:, None, :] + basis[None]) * a).reshape(-1, 3)
    m = np.full(len(pos), configs.ARGON["mass"])
    (name, _, top), = wl.species
    wl = dataclasses.replace(wl, species=[(name, len(pos), top)], pos=pos, mass_amu=m, box=a * max(nx, ny, nz),
                             vel=configs.maxwell_boltzmann(m, 120.0, np.random.default_rng(seed)))
    sysm = build_system(shaken(wl, seed))
    sysm["hmat"] = np.diag([nx * a, ny * a, nz * a])
    return sysm


def binary(n, seed=5):
    return build_system(shaken(configs.lj_box(n, 0.75, 1.0, seed, charged=True), seed))


CASES = {
    "water-375 (1 or 2 cells)": lambda: water(5),
    "water-648": lambda: water(6),
    "water-3000 (2 cells, no staging)": lambda: water(10),
    "water-3993 (3 cells)": lambda: water(11),
    "water-5184, skin 1.5": lambda: water(12, 1.5),
    "water-8232": lambda: water(14),
    "slab 3 x 6 x 9": lambda: slab(3, 6, 9),
    "slab 4 x 4 x 12": lambda: slab(4, 4, 12),
    "argon-64": lambda: build_system(shaken(configs.lj_box(64, 0.8, 1.0, 2), 2)),
    "argon-1372": lambda: slab(7, 7, 7),
    "binary-100": lambda: binary(100),
    "binary-2047 odd": lambda: binary(2047),
}


def pair_keys(i, j, n):
    """the pairs as sorted keys, whichever atom comes first"""
    return np.sort(np.minimum(i, j).astype(np.int64) * n + np.maximum(i, j))


def forces(sysm, mode, monkeypatch, walk=False):
    if walk:
        monkeypatch.setenv("CM3D_NB_LIST_KERNEL", "walk")
    e = Engine(sysm, mode=mode)
    if walk:
        monkeypatch.delenv("CM3D_NB_LIST_KERNEL")
    e.get_ngbr()
    e.force(1)
    f = e.forces(_abi.FXL)
    st = e.status()
    lists = [e.pair_list(w) for w in range(4)]
    e.close()
    assert st["nonfinite"] == 0 and st["stage_timeouts"] == 0
    return f, lists


@pytest.mark.parametrize("name", list(CASES))
def test_lists_of_every_grid(engine_lib, name, monkeypatch):
    sysm = CASES[name]()
    n = sysm.natoms
    orc = Oracle(sysm)
    orc.get_ngbr()
    f, lists = forces(sysm, _abi.MIXED, monkeypatch)
    fw, _ = forces(sysm, _abi.MIXED, monkeypatch, walk=True)
    fp, plists = forces(sysm, _abi.PLAIN_FP64, monkeypatch)
    for w in range(4):
        want = pair_keys(*orc.pair_list(w), n)
        for i, j in (lists[w], plists[w]):
            np.testing.assert_array_equal(pair_keys(i, j, n), want)
    np.testing.assert_array_equal(f, fw)
    assert rel_rms(f, fp) <= 1e-5
