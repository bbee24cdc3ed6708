"""x | y | z blocks that lie back to back but are not page-locked as one: pageable, one of three page-locked, each
page-locked by itself, all in one piece.  Every copy in and out must be what the arrays hold."""
import mmap

import numpy as np
import pytest

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system

pytestmark = pytest.mark.gpu

N = 2048                                       # a block of whole pages
# the page-locked ranges, in blocks
LOCKED = {"none": [], "first": [(0, 1)], "middle": [(1, 2)], "last": [(2, 3)], "one by one": [(0, 1), (1, 2), (2, 3)],
          "first two, last": [(0, 2), (2, 3)], "whole": [(0, 3)]}


@pytest.mark.parametrize("name", list(LOCKED))
def test_blocks_back_to_back(engine_lib, name):
    import torch
    rt = torch.cuda.cudart()
    sysm = build_system(configs.lj_box(N, 1.0, 1.0, 4))
    assert sysm.natoms == N and 8 * N % mmap.PAGESIZE == 0
    block = mmap.mmap(-1, 3 * 8 * N)
    a = np.frombuffer(block, dtype=np.float64).reshape(3, N)
    with Engine(sysm, mode=_abi.MIXED) as e:
        locked = []
        try:
            for b0, b1 in LOCKED[name]:
                at = a.ctypes.data + 8 * N * b0
                assert int(rt.cudaHostRegister(at, 8 * N * (b1 - b0), 0)) == 0
                locked.append(at)
            e.step_init()
            for put, get in ((e.set_positions, e.positions), (e.set_velocities, e.velocities),
                             (e.set_forces, e.forces)):
                want = np.random.default_rng(3).normal(size=(3, N))
                a[:] = want
                put(a)
                np.testing.assert_array_equal(get(), want)       # a pageable array of its own
                a[:] = 0.0
                get(out=a)
                np.testing.assert_array_equal(a, want)
        finally:
            for at in locked:
                assert int(rt.cudaHostUnregister(at)) == 0
