"""A list that outgrows its slots in a replayed step halts the step while other blocks of the list kernel start and the
k-space runs beside it; the host then widens the slots and finishes the step.  The step must end as the host-driven one
does, and no block may be split by the halt: threads that share descriptors through shared memory leave together."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT, rel_rms
from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system

CSRC = os.path.join(ROOT, "cm3d_b200", "csrc")
COOPERATE = re.compile(r"__shared__|__syncthreads|__shfl|__ballot|sys_acc|block_acc|split_sum|warp_sum|warp_totals|"
                       r"cw_convert_atom|full_list_atom|walk_candidates")


def kernels(name):
    """(kernel, its parameters, its body) of a source file"""
    with open(os.path.join(CSRC, name)) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*(?:\([^)]*\))?[^)]*\)\s*)?(\w+)\s*\(", text):
        level, k = 1, m.end()
        while level:
            level += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        head, b = text[m.end():k - 1], text.index("{", k)
        level, k = 1, b + 1
        while level:
            level += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), head, text[b:k]


def test_blocks_leave_together():
    """Every kernel that raises the halt, and every kernel that runs beside those, takes its gate for the whole block
    where its threads work together."""
    seen = set()
    for name in ("nb_list.cu", "nb_cwin.cu", "nb_kspace.cu", "nb_step.cu"):
        for kernel, head, body in kernels(name):
            beside = name == "nb_kspace.cu" or kernel in ("k_group_init", "k_group_small")
            if not (beside or re.search(r"\bhalt\b", head)) or not COOPERATE.search(body):
                continue
            if "gated_off(" not in body:
                continue                              # a kernel of host-driven calls
            seen.add(kernel)
            assert not re.search(r"(?<!block_)\bgated_off\(", body), kernel
            # the first thing the kernel does: every thread of the block is there
            assert re.match(r"\{\s*if \(block_gated_off\(", body), kernel
    assert {"k_list_tile", "k_list_win", "k_list_full", "k_list_half", "k_cw_convert", "k_sfac_gemm", "k_kforce_reg",
            "k_kforce_mixed", "k_sfac_mixed", "k_sred", "k_group_small"} <= seen


# ------------------------------------------------------------------- on the GPU
def stretched(wl, per, times):
    """The workload in a box `times` as long along z, and two sets of positions: its groups of `per` atoms spread evenly
    over the box, and all of them in its lowest part -- with lists beyond their slots' room, 1.3 times the mean and 64
    entries, to the next multiple of 32."""
    sysm = build_system(wl)
    dense = np.stack([sysm["px"], sysm["py"], sysm["pz"]]).astype(float)
    spread = dense.copy()
    spread[2] += (times - 1) * np.repeat(dense[2, ::per], per)
    sysm["hmat"] = np.diag([wl.box, wl.box, times * wl.box])
    sysm["px"], sysm["py"], sysm["pz"] = spread
    return sysm, dense


def water_large_sum():
    return [stretched(configs.water_box(ngrid=16, seed=2, alpha=0.31, kmax=13, placement="octant"), 3, 2)]


def argon():
    return [stretched(configs.lj_box(4000, 1.0, 1.0, 4), 1, 10)]


def staged_batch():
    return [stretched(configs.lj_box(2048, 1.0, 1.0, 4), 1, 10)] * 80


def charged_batch():
    return [stretched(configs.lj_box(n, 1.0, 1.0, n, charged=True), 1, 10) for n in (1000, 2047)]


@pytest.mark.gpu
@pytest.mark.parametrize("make", [water_large_sum, argon, staged_batch, charged_batch])
def test_a_halted_step_ends_as_the_host_driven_one(engine_lib, make):
    parts = make()
    systems, dense = [p[0] for p in parts], np.concatenate([p[1] for p in parts], axis=1)
    out = []
    for graph in (True, False):
        e = Engine(systems if len(systems) > 1 else systems[0], mode=_abi.MIXED, use_graph=graph)
        e.step_init()
        e.step(1, 1)
        e.set_positions(dense)
        e.step(100, 2)
        out.append((e.positions(), e.velocities(), e.forces(_abi.FXL), e.status(), e.energies_table()))
        e.close()
    (pos, vel, f, st, en), (pos2, vel2, f2, st2, en2) = out
    assert st["overflows"] > st2["overflows"]
    assert st["nonfinite"] == 0 and st["stage_timeouts"] == 0
    # the same lists; the forces' partial sums are added in another order
    np.testing.assert_allclose(pos, pos2, rtol=0, atol=1e-9)
    assert rel_rms(vel, vel2) <= 1e-9
    assert rel_rms(f, f2) <= 1e-6
    for k in ("vinter", "velec", "vewald"):
        np.testing.assert_allclose(en[k], en2[k], rtol=1e-7, atol=1e-7 * np.abs(en2["poter"]).max())
