"""The staged list kernel on both sides of its rule: even batches from 400 atoms per SM, ragged ones from 1024, and one
large box.  The lists, seen through the forces, are bit for bit those of the warp-per-atom walk."""
import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from test_list_kernels import binary, shaken

pytestmark = pytest.mark.gpu


def lj(n, seed=7):
    return build_system(shaken(configs.lj_box(n, 0.8, 1.0, seed), seed))


CASES = {
    "even, 61,440": lambda: [lj(2048)] * 30,
    "even, 57,344 (walked)": lambda: [lj(2048)] * 28,
    "even, charged, 69,598": lambda: [binary(2047)] * 34,
    "ragged, 64,016 (walked)": lambda: [lj(108)] * 188 + [lj(1372, 3)] * 32,
    "one box, 62,500": lambda: lj(62500),
}


@pytest.mark.parametrize("name", list(CASES))
def test_staged_and_walked(engine_lib, name, monkeypatch):
    system = CASES[name]()
    out = []
    for walk in (False, True):
        if walk:
            monkeypatch.setenv("CM3D_NB_LIST_KERNEL", "walk")
        with Engine(system, mode=_abi.MIXED) as e:
            e.get_ngbr()
            e.force(1)
            out.append(e.forces(_abi.FXL))
            assert e.status()["nonfinite"] == 0
    np.testing.assert_array_equal(out[0], out[1])
