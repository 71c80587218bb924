"""The tissue guard in automatic mode (bricks) on the smallest lattices, against the whole-GPU frame and
the oracle bit for bit."""
import ctypes as ct

import numpy as np
import pytest

from genesis_tissue_simulation_gb300 import workloads as W
from genesis_tissue_simulation_gb300.grid import build_grid
from genesis_tissue_simulation_gb300.native_backend import Capsule, GraspParams, PlainTissue, pointer

pytestmark = pytest.mark.gpu
GRASP = dict(W.DEFAULT_GRASP, ccd_velocity=0.0)


def block(size):
    return build_grid(0.2, size=tuple(np.float64(c) * 0.2 - 0.02 for c in size), density=1000.0)


def arm_guard(t, minimum=0.5, passes=1):
    t.check("LCS_SetTissueGuard", ct.c_float(minimum), passes, len(t.grid.positions), pointer(t.grid.inside), 1)
    t.check("LCS_SetTissueMaterial", ct.c_float(80.0), ct.c_float(0.01))


def press(t, k, steps=5):
    """Capsule across the top face of the block, lower every frame."""
    nodes = t.grid.positions[t.grid.active != 0]
    top, mid = float(nodes[:, 1].max()), nodes.mean(axis=0)
    y = top + 0.2 - 0.2 * (k + 1) / steps
    t.set_capsule(Capsule((mid[0] - 1.0, y, mid[2]), (mid[0] + 1.0, y, mid[2]), 0.25))


def guarded(lib, size, mode, steps=5):
    with PlainTissue(block(size), dt=1 / 60, substeps=6, ks=1e6, strain_damping_s=0.0, grasp_params=GraspParams(**GRASP), dll_path=lib) as t:
        try:
            if mode is not None:
                assert t.dll.LCS_SetLaunchMode(mode) == 0
            t.set_gravity(0.0, -981.0, 0.0)
            arm_guard(t)
            frames = []
            for k in range(steps):
                press(t, k, steps)
                t.step()
                frames.append((t.positions(), t.velocities()))
            return frames
        finally:
            if mode is not None:
                t.dll.LCS_SetLaunchMode(0)


# CTAs of one warp (up to 64 nodes) and of more
@pytest.mark.parametrize("size", [(2, 2, 2), (3, 3, 3), (4, 2, 3), (3, 3, 4), (7, 4, 5)])
def test_guarded_small_lattices_match_the_whole_gpu_frame_and_the_oracle(gpu_lib, oracle_libs, size):
    got = guarded(gpu_lib, size, 0)
    for want in (guarded(gpu_lib, size, 1), guarded(oracle_libs[0], size, None)):
        for k, (a, b) in enumerate(zip(got, want)):
            assert np.isfinite(b[0]).all()
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), k
