"""The tissue guard armed after frames have run: its frames follow the current topology (severed links,
and without edge stiffness the edges that live tets carry), in automatic mode as on the whole GPU."""
import ctypes as ct

import numpy as np
import pytest

from test_guard_bricks import GRASP, arm_guard, block, press
from genesis_tissue_simulation_gb300.native_backend import GraspParams, PlainTissue, blade_sweep

pytestmark = pytest.mark.gpu


def late_guard(lib, mode, ks, sever, no_alloc):
    with PlainTissue(block((9, 6, 7)), dt=1 / 60, substeps=5, ks=ks, strain_damping_s=0.04, grasp_params=GraspParams(**GRASP), dll_path=lib) as t:
        try:
            assert t.dll.LCS_SetLaunchMode(mode) == 0
            step = t.dll.LCS_StepNoAlloc if no_alloc else t.dll.LCS_Step
            step.argtypes, step.restype = (ct.c_float,), ct.c_int
            t.set_gravity(0.0, -981.0, 0.0)
            nodes = t.grid.positions[t.grid.active != 0]
            top, mid = float(nodes[:, 1].max()), nodes.mean(axis=0)
            for k in range(3):
                press(t, k)
                if sever and k == 1:
                    t.set_blade(blade_sweep((mid[0] + 0.02, top + 1.0, mid[2] - 0.4), (mid[0] + 0.02, mid[1], mid[2] - 0.4),
                                            (mid[0] + 0.02, top + 1.0, mid[2] + 0.4), (mid[0] + 0.02, mid[1], mid[2] + 0.4)))
                assert step(t.dt) == 0
                if sever and k == 1:
                    t.check("LCS_DetectCut")
                    t.functions["LCS_SetPressureCutMode"](1)   # plain frames of a severed lattice follow
            if not no_alloc:   # the guard may be armed again once the stiffnesses are new
                t.set_tet_stiffness(*t.tet_stiffness())
            arm_guard(t)
            out = [t.neighbors()]
            for k in range(3, 6):
                press(t, k)
                assert step(t.dt) == 0
                out += [t.positions(), t.velocities()]
            return t.grid, out
        finally:
            t.dll.LCS_SetLaunchMode(0)


@pytest.mark.parametrize("no_alloc", [False, True], ids=["step", "no-alloc"])
@pytest.mark.parametrize("ks,sever", [(1e6, True), (0.0, False), (0.0, True)], ids=["severed", "fallback", "severed-fallback"])
def test_a_guard_armed_after_frames_follows_the_topology(gpu_lib, ks, sever, no_alloc):
    grid, got = late_guard(gpu_lib, 0, ks, sever, no_alloc)
    _, want = late_guard(gpu_lib, 1, ks, sever, no_alloc)
    assert not sever or (want[0] != grid.neighbors).sum() > 0
    for a, b in zip(got, want):
        assert np.isfinite(b).all() and np.array_equal(a, b)
