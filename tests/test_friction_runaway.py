"""Contact model 1 on a state that has flown apart: the sweep of a node against an instrument ends, with the
speed of a node's path infinite in float (the steps of the conservative advancement are zero) or merely huge."""
import ctypes as ct
import multiprocessing as mp

import numpy as np
import pytest

from genesis_tissue_simulation_gb300.native_backend import GraspParams, PlainTissue, pointer
from test_friction_contact import grasper
from test_guard_bricks import GRASP, block


def runaway(lib, speed, mode=None, substeps=2):
    with PlainTissue(block((4, 3, 4)), dt=1 / 60, substeps=substeps, ks=1e6, strain_damping_s=0.0, grasp_params=GraspParams(**GRASP), dll_path=lib) as t:
        try:
            if mode is not None:
                assert t.dll.LCS_SetLaunchMode(mode) == 0
            t.check("LCS_SetContactModel", 1, ct.c_float(0.6), ct.c_float(0.4), ct.c_float(0.1), ct.c_float(0.01))
            top = float(t.grid.positions[t.grid.active != 0, 1].max())
            for k in (0, 1):
                t.check("LCS_SetGraspTool", ct.byref(grasper(top, k, 4, True)))
            vel = np.tile(np.float32([speed, 0.3 * speed, -0.2 * speed]), (len(t.grid.positions), 1))
            assert t.dll.GBT_SetState(None, pointer(vel), None, None, None, None, None, None, 0, 0) == 0
            t.step()
            return t.positions()
        finally:
            if mode is not None:
                t.dll.LCS_SetLaunchMode(0)


def _oracle(lib, speed, out):
    out.put(runaway(lib, speed).shape)


@pytest.mark.parametrize("speed", [1e6, 1e12, 1e23])
def test_the_oracle_leaves_a_runaway_state(oracle_libs, speed):
    context = mp.get_context("spawn")
    out = context.Queue()
    worker = context.Process(target=_oracle, args=(str(oracle_libs[0]), speed, out))
    worker.start()
    worker.join(60)
    ended = not worker.is_alive()
    if not ended:
        worker.kill()
    assert ended and worker.exitcode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("speed", [1e6, 1e12, 1e23])
def test_frames_leave_a_runaway_state(gpu_lib, oracle_libs, speed, mode):
    got, want = runaway(gpu_lib, speed, mode), runaway(oracle_libs[0], speed)
    assert np.array_equal(got, want, equal_nan=True)
