"""The admission estimate bounds what a job's context takes: against memory measured on a B200 (CPU), and against the
device's own account of it on the GPU."""
import math

import numpy as np
import pytest

from cm3d_b200 import configs
from cm3d_b200.serving import device_bytes
from cm3d_b200.setup import build_system


class Cube(dict):
    """the fields device_bytes reads of a water box: cut-off 10 A, skin `skin`, every atom charged"""

    def __init__(self, ngrid, skin, ktot):
        L = ngrid * configs.WATER_SPACING
        rl = 10.0 + skin
        super().__init__(hmat=np.diag([L, L, L]).ravel(), rmaxl_skin2=np.array([rl * rl]), ninter=1, ktot=ktot,
                         rmaxl_skin2_e=rl * rl, skin=skin)
        self.natoms = 3 * ngrid ** 3


# molecules an edge, skin, k-vectors, bytes that create, step_init and three steps took
@pytest.mark.parametrize("ngrid,skin,ktot,used", [
    (14, 0.5, 709, 56.6e6), (16, 0.5, 1054, 98.6e6), (20, 0.5, 1535, 180.4e6), (24, 0.5, 2787, 314.6e6),
    (33, 0.5, 7073, 824.2e6), (48, 1.5, 19455, 2669.7e6)])
def test_estimate_bounds_what_was_measured(ngrid, skin, ktot, used):
    assert used <= device_bytes(Cube(ngrid, skin, ktot)) <= 1.5 * used


def water(ngrid, kmax):
    return build_system(configs.water_box(ngrid=ngrid, seed=2, kmax=kmax, placement="octant"))


def binary(n):
    return build_system(configs.lj_box(n, 0.8, 1.0, 4, charged=True))


@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda: water(8, 2), lambda: water(16, 7), lambda: water(16, 13), lambda: water(22, 12),
                                  lambda: binary(9826), lambda: build_system(configs.lj_box(32000, 0.8, 1.0, 4))],
                         ids=["water-1536", "water-12288", "water-12288 large sum", "water-31944 large sum",
                              "binary-9826", "argon-32000"])
def test_estimate_bounds_what_a_context_takes(engine_lib, make):
    import torch
    from cm3d_b200.engine import Engine

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    system = make()
    with Engine(binary(200)) as e:                    # the context and its module are not the job's
        e.step_init()
        e.step(1, 2)
    before = used()
    with Engine(system) as e:
        e.step_init()
        e.step(1, 2)
        took = used() - before
    assert took <= device_bytes(system)
    assert math.isfinite(took)
