"""Automatic mode where frames cannot run on bricks (bends, perpendicular damping, a guard with two passes): the
session makes no plan it would not use, and the frames timed in one CTA, on the whole GPU and on one cluster
(the 2nd to 4th) and those in the shape that was kept give the whole-GPU frames bit for bit."""
import ctypes as ct

import numpy as np
import pytest

from genesis_tissue_simulation_gb300.native_backend import GraspParams, PlainTissue
from test_guard_bricks import GRASP, arm_guard, block, press

pytestmark = pytest.mark.gpu


def frames(lib, size, mode, guard_passes=0, steps=7, **material):
    with PlainTissue(block(size), dt=1 / 60, substeps=4, ks=1e6, strain_damping_s=0.04, grasp_params=GraspParams(**GRASP), dll_path=lib, **material) as t:
        try:
            assert mode is None or t.dll.LCS_SetLaunchMode(mode) == 0
            t.set_gravity(0.0, -981.0, 0.0)
            if guard_passes:
                arm_guard(t, passes=guard_passes)
            info = np.zeros(4, np.int32)
            assert mode is None or t.dll.GBT_BrickInfo(info.ctypes.data_as(ct.c_void_p)) == 0
            out = []
            for k in range(steps):
                press(t, k, steps)
                t.step()
                out.append((t.positions(), t.velocities(), t.bend_alive()))
            return out, int(info[0])
        finally:
            if mode is not None:
                t.dll.LCS_SetLaunchMode(0)


@pytest.mark.parametrize("size", [(4, 3, 3), (11, 6, 9)])   # fits one CTA, and one cluster
@pytest.mark.parametrize("options", [dict(kb=1e2, cb=1e-3), dict(cs=1e-3), dict(guard_passes=2)], ids=["bends", "perpendicular", "guard-2"])
def test_automatic_mode_without_bricks_matches_the_whole_gpu(gpu_lib, size, options):
    got, bricks = frames(gpu_lib, size, 0, **options)
    want, _ = frames(gpu_lib, size, 1, **options)
    assert bricks == 0 or "guard_passes" in options
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.isfinite(b[0]).all()
        for x, y in zip(a, b):
            assert np.array_equal(x, y), k


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("size", [(4, 3, 3), (11, 6, 9)])
def test_perpendicular_damping_matches_the_oracle(gpu_lib, oracle_libs, size, mode):
    """A damping pass ends with every node's velocity scaled and the next substep's predict takes the nodes in
    another order, in every shape."""
    got, _ = frames(gpu_lib, size, mode, cs=1e-3, alpha=0.5)
    want, _ = frames(oracle_libs[0], size, None, cs=1e-3, alpha=0.5)
    for k, (a, b) in enumerate(zip(got, want)):
        assert np.isfinite(b[0]).all()
        for x, y in zip(a, b):
            assert np.array_equal(x, y), k
