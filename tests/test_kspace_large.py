"""Reciprocal space of one system by the large-sum kernels (k_sfac_gemm, k_kforce_reg): k sets around the sizes of
their register and tile groups (|kc| 8, 12, 16, 21, 24), atom counts that leave ragged tiles, a k list that is not
CM3D's symmetric one (rows cut on one side, gaps), and two that stay with the older kernels (too small a sum, too large
a |kc|), against the plain FP64 engine on the same positions.

Tolerances: the mixed engine's (level-1 forces 1e-5 relative RMS, energies 1e-5, virials 5e-5).  Two evaluations on the
same positions give the same bits."""
import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi, configs, engine
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system

pytestmark = pytest.mark.gpu


def water(ngrid, kmax):
    base = configs.water_box(ngrid=ngrid, seed=3, alpha=0.31, kmax=kmax, placement="octant")
    return build_system(base)


def thin(sysm, keep):
    """the system with only the k-vectors keep(ka, kb, kc) of its set"""
    k = np.stack([sysm["ka"], sysm["kb"], sysm["kc"]])
    k = k[:, keep(*k)]
    for name, v in zip(("ka", "kb", "kc"), k):
        sysm[name] = v
    sysm["ktot"] = k.shape[1]
    return sysm


CASES = {
    "kmax 12, 12288": lambda: water(16, 12),
    "kmax 13, 12288": lambda: water(16, 13),
    "kmax 16, 6591": lambda: water(13, 16),
    "kmax 17, 6591": lambda: water(13, 17),
    "kmax 21, 5184": lambda: water(12, 21),
    "kmax 24, 3993": lambda: water(11, 24),
    "kmax 8, 41472": lambda: water(24, 8),
    "one-sided rows": lambda: thin(water(16, 16), lambda a, b, c: (c > -9) & ((a + b) % 3 != 1)),
    "gaps along kc": lambda: thin(water(16, 16), lambda a, b, c: (c % 5 != 2) & (np.abs(c) < 13)),
    "kmax 25: the older kernels": lambda: water(11, 25),
}


@pytest.mark.parametrize("name", list(CASES))
def test_large_sums(engine_lib, name):
    sysm = CASES[name]()
    out = []
    for mode in (_abi.MIXED, _abi.PLAIN_FP64):
        with Engine(sysm, mode=mode) as e:
            e.get_ngbr()
            runs = []
            for _ in range(2):
                e.force(1)
                runs.append(e.forces(_abi.FXL))
            if mode == _abi.MIXED:
                np.testing.assert_array_equal(runs[0], runs[1])
            out.append((runs[0], e.getvewald()))
    (f, v), (fp, vp) = out
    assert rel_rms(f, fp) <= 1e-5
    assert abs(v["vewald"] - vp["vewald"]) <= 1e-5 * abs(vp["vewald"])
    t = np.abs(vp["wewaldtensor"]).max()
    np.testing.assert_allclose(v["wewaldtensor"], vp["wewaldtensor"], rtol=0, atol=5e-5 * t)
