"""Without memory for the brick tables a session, its guard, a rollout and a batch open all the same and run in
the other launch shapes.  The failing allocation is a stand-in of the debug build."""
import ctypes as ct

import numpy as np
import pytest

from genesis_tissue_simulation_gb300 import batch as BT
from genesis_tissue_simulation_gb300 import diff as DF
from genesis_tissue_simulation_gb300.native_backend import GraspParams, PlainTissue
from test_debug_bounds import debug_lib  # noqa: F401  (fixture)
from test_guard_bricks import GRASP, arm_guard, block, press

pytestmark = pytest.mark.gpu
SIZE = (7, 5, 6)


def fail(lib, count):
    assert ct.CDLL(str(lib)).GBT_DebugFailBrickTables(count) == 0


def session(lib, refusals, guard_refusals=None, mode=0):
    fail(lib, refusals)
    try:
        with PlainTissue(block(SIZE), dt=1 / 60, substeps=4, ks=1e6, strain_damping_s=0.0, grasp_params=GraspParams(**GRASP), dll_path=lib) as t:
            fail(lib, 0)
            try:
                assert t.dll.LCS_SetLaunchMode(mode) == 0
                info = np.zeros(4, np.int32)
                assert t.dll.GBT_BrickInfo(info.ctypes.data_as(ct.c_void_p)) == 0
                if guard_refusals is not None:
                    fail(lib, guard_refusals)
                    arm_guard(t)
                    fail(lib, 0)
                t.set_gravity(0.0, -981.0, 0.0)
                for k in range(3):
                    press(t, k)
                    t.step()
                return t.positions(), int(info[0])
            finally:
                t.dll.LCS_SetLaunchMode(0)
    finally:
        fail(lib, 0)


@pytest.mark.parametrize("guard", [False, True])
def test_sessions_open_without_memory_for_bricks(debug_lib, guard):  # noqa: F811
    got, bricks = session(debug_lib, 0 if guard else 1, 1 if guard else None)
    want, _ = session(debug_lib, 0, 0 if guard else None, mode=1)
    assert (bricks > 0) == guard and np.array_equal(got, want)


def test_rollouts_open_without_memory_for_bricks(debug_lib):  # noqa: F811
    import torch
    out = []
    for refusals in (0, 1):
        with DF.DifferentiableTissue(block(SIZE), dt=1 / 60, substeps=4, ks=1e6, gravity=(0.0, -981.0, 0.0), checkpoint_every=3, max_frames=2,
                                     dll_path=debug_lib, scale_modulus=1e6) as t:
            # the session has its plan; the reverse sweep's is made here again, with or without memory
            fail(debug_lib, refusals)
            try:
                t._check("GBT_DiffBegin", 1e6, 3, 2)
            finally:
                fail(debug_lib, 0)
            theta = torch.full((t.tet_count,), float(np.log(1e-6)), device="cuda")
            x = t.forward(theta, None, frames=2)
            out.append((x.cpu().numpy(), t.backward(torch.ones_like(x))["theta"].cpu().numpy(), t.info()["ctas"]))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-6 * np.abs(out[0][1]).max()


def test_batches_open_without_memory_for_bricks(debug_lib):  # noqa: F811
    out = []
    for refusals in (0, 1):
        fail(debug_lib, refusals)
        try:
            with BT.TissueBatch([block((3, 3, 4)), block((5, 3, 3))], dt=1 / 60, substeps=3, ks=1e6, grasp_params=GraspParams(**GRASP),
                                dll_path=debug_lib) as b:
                b.set_gravity(0.0, -981.0, 0.0)
                for _ in range(3):
                    b.step()
                out.append(b.positions())
        finally:
            fail(debug_lib, 0)
    assert np.array_equal(out[0], out[1])
