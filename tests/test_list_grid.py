"""The engine's own list radius against the compact pair kernel: wider lists make wider cells, and a window of 27 of them
has to fit beside the tables.  Water boxes (skin 0.5 or 1 A, cut-off 10 A) whose grid by CM3D's radius holds such windows
and whose grid by the full list skin does not: the skin stops where the kernel would be lost, and is taken in full where
that would leave less than a tenth of the cut-off.  Either way the lists hold every pair: the forces are the plain FP64
engine's to the mixed engine's bound (1e-5 relative RMS)."""
import numpy as np
import pytest

from conftest import rel_rms
from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system
from test_list_kernels import shaken

pytestmark = pytest.mark.gpu


def water(ngrid, skin):
    return build_system(shaken(configs.water_box(ngrid=ngrid, seed=ngrid, rc=10.0, alpha=0.31, kmax=3, skin=skin,
                                                 placement="octant"), 1, 0.02))


def level1(sysm, mode):
    with Engine(sysm, mode=mode) as e:
        e.get_ngbr()
        e.force(1)
        systems = range(len(sysm) if isinstance(sysm, list) else 1)
        return e.forces(_abi.FXL), e.pair_kernel()[0], [e.grid(s)[0][0] for s in systems]


# molecules an edge, skin, cells an edge, compact kernel
@pytest.mark.parametrize("ngrid,skin,cells,compact", [
    (16, 0.5, 4, True),     # the full skin, windows beside eight copies of the erfc tables
    (18, 0.5, 4, True),     # the full skin, windows beside four copies
    (21, 0.5, 5, True),
    (18, 1.5, 4, True),
    (15, 0.5, 4, True),     # 3 cells by the full skin, too wide beside four copies; 1.6 A of skin with 4
    (15, 1.0, 4, True),
    (14, 0.5, 3, False),    # 0.86 A of skin with 4 cells: the full skin instead
])
def test_skin_and_compact_kernel(engine_lib, ngrid, skin, cells, compact):
    sysm = water(ngrid, skin)
    f, kernel, grid = level1(sysm, _abi.MIXED)
    assert grid == [cells]
    assert (kernel == "compact") == compact
    assert rel_rms(f, level1(sysm, _abi.PLAIN_FP64)[0]) <= 1e-5


@pytest.mark.parametrize("sizes,cells", [([14, 11, 15], [4, 3, 4]), ([11, 18], [3, 4])])
def test_a_batch_keeps_its_compact_kernel(engine_lib, sizes, cells):
    """one system of a batch must not take the kernel from the others"""
    systems = [water(n, 0.5) for n in sizes]
    f, kernel, grid = level1(systems, _abi.MIXED)
    assert kernel == "compact"
    assert grid == cells
    fp = np.concatenate([level1(s, _abi.PLAIN_FP64)[0] for s in systems], axis=1)
    assert rel_rms(f, fp) <= 1e-5
