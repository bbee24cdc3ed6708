"""Which reciprocal-space kernels run, on both sides of the rule (charges times k-vectors from 5e7, |kc| up to 24), seen
in the launches of one evaluation (seven by the large-sum kernels, five by the older ones); k sets that reach each
register size of the force kernel (|kc| up to 8, 12, 16, 24), against the plain FP64 engine to the mixed engine's bounds
(forces 1e-5 relative RMS, energy 1e-5, virial 5e-5)."""
import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi
from cm3d_b200.engine import Engine
from test_kspace_large import thin, water

pytestmark = pytest.mark.gpu

CASES = {
    # the system, the large-sum kernels' side
    "kmax 12, 14739": (lambda: water(17, 12), True),
    "|kc| 8 of kmax 16, 10125": (lambda: thin(water(15, 16), lambda a, b, c: np.abs(c) <= 8), True),
    "|kc| 1 of kmax 24, 31944": (lambda: thin(water(22, 24), lambda a, b, c: np.abs(c) <= 1), True),
    "kmax 13, 12288": (lambda: water(16, 13), True),
    "kmax 17, 6591": (lambda: water(13, 17), True),
    "kmax 12, 12288, too small a sum": (lambda: water(16, 12), False),
    "kmax 25, 3993, too large a |kc|": (lambda: water(11, 25), False),
}


@pytest.mark.parametrize("name", list(CASES))
def test_kernels_of_each_side(engine_lib, name):
    make, large = CASES[name]
    sysm = make()
    assert large == (sysm.natoms * sysm["ktot"] >= 5e7 and np.abs(sysm["kc"]).max() <= 24)
    out = []
    for mode in (_abi.MIXED, _abi.PLAIN_FP64):
        with Engine(sysm, mode=mode) as e:
            e.get_ngbr()
            e.fk_ewald()
            if mode == _abi.MIXED:
                before = e.launch_count()
                e.fk_ewald()
                assert (e.launch_count() - before == 7) == large
            e.force(1)
            out.append((e.forces(_abi.FXL), e.getvewald()))
    (f, v), (fp, vp) = out
    assert rel_rms(f, fp) <= 1e-5
    assert abs(v["vewald"] - vp["vewald"]) <= 1e-5 * abs(vp["vewald"])
    t = np.abs(vp["wewaldtensor"]).max()
    np.testing.assert_allclose(v["wewaldtensor"], vp["wewaldtensor"], rtol=0, atol=5e-5 * t)
