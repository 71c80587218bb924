"""The debug build's index checks in automatic mode, where frames run on bricks: local nodes of elements, nodes,
exchange records and colour slots of sessions (plain, capsule, blade, guard, friction, adapter settings), rollouts
and batches.  No index is out of range, the bricks did check (their count says so), and the checks leave the
results alone."""
import ctypes as ct

import numpy as np
import pytest

from genesis_tissue_simulation_gb300 import batch as BT
from genesis_tissue_simulation_gb300 import build as native_build
from genesis_tissue_simulation_gb300 import workloads as W
from genesis_tissue_simulation_gb300.native_backend import GraspParams, PlainTissue
from test_debug_bounds import SMALL, _read, _run, debug_lib  # noqa: F401  (fixture)
from test_guard_bricks import GRASP, block, press


def checks(dll, name="GBT_DebugBrickChecks"):
    out = ct.c_uint(0)
    assert getattr(dll, name)(ct.byref(out)) == 0
    return out.value


def test_release_build_counts_nothing():
    dll = ct.CDLL(str(native_build.build()))
    out = ct.c_uint(0)
    assert dll.GBT_DebugBrickChecks(ct.byref(out)) == -4001 and dll.GBT_BatchDebugBrickChecks(ct.byref(out)) == -4001
    assert dll.GBT_DebugFailBrickTables(1) == -4001


def sound(session, name=""):
    record = _read(session.dll)
    assert record[0] == 0, f"{record[0]} out-of-range gathers, first index {record[1]} at site {record[2]}"
    assert checks(session.dll) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("name,scale,steps", [("c1", None, 6), ("c2", SMALL, 8), ("c3", SMALL, 12)])
def test_workloads_on_bricks(gpu_lib, debug_lib, name, scale, steps):  # noqa: F811
    w = W.make(name, steps=steps, scale=scale)
    s = w.open(debug_lib)
    try:
        s.dll.LCS_SetLaunchMode(0)
        w.run(s, steps=steps)
        sound(s)
        got = s.positions()
    finally:
        s.close()
    assert np.array_equal(got, _run(w, gpu_lib, steps)[0])


@pytest.mark.gpu
def test_guard_and_friction_on_bricks(debug_lib):  # noqa: F811
    from test_friction_contact import friction_run
    from test_guard import guarded_run
    guarded_run(debug_lib, steps=4, launch_mode=0, on_close=sound)
    friction_run(debug_lib, steps=4, closing=True, launch_mode=0, on_close=sound)


@pytest.mark.gpu
@pytest.mark.parametrize("size,bricks", [((2, 2, 2), 0), ((9, 6, 13), 27), ((17, 3, 11), 152)])
def test_damped_sessions_without_edge_stiffness_on_bricks(debug_lib, size, bricks):  # noqa: F811
    dll = ct.CDLL(str(debug_lib))
    assert dll.GBT_SetBrickCount(bricks) == 0
    try:
        with PlainTissue(block(size), dt=1 / 60, substeps=4, ks=0.0, strain_damping_s=0.04, grasp_params=GraspParams(**GRASP), dll_path=debug_lib) as t:
            t.dll.LCS_SetLaunchMode(0)
            t.set_gravity(0.0, -981.0, 0.0)
            for k in range(3):
                press(t, k)
                t.step()
            sound(t)
    finally:
        dll.GBT_SetBrickCount(0)


@pytest.mark.gpu
@pytest.mark.parametrize("bricks", [1, 7, 0])
def test_rollouts_on_bricks(debug_lib, bricks):  # noqa: F811
    import torch

    from diff_cases import Case
    from test_gpu_adjoint import gpu_tissue
    case = Case()
    dll = ct.CDLL(str(debug_lib))
    assert dll.GBT_SetBrickCount(bricks) == 0
    try:
        with gpu_tissue(case, debug_lib, 0) as t:
            x = t.forward(torch.tensor(case.theta(t.session.tet_count), device="cuda"), torch.tensor(case.path, device="cuda"))
            sound(t.session)
            grads = t.backward(torch.ones_like(x), rest_shape=True)
            assert torch.isfinite(grads["theta"]).all()
            sound(t.session)
    finally:
        dll.GBT_SetBrickCount(0)


@pytest.mark.gpu
@pytest.mark.parametrize("count", [3, 160])   # spread over several CTAs, several to a CTA
def test_batches_on_bricks(debug_lib, count):  # noqa: F811
    wl = BT.make_c4(count=count, seed=11, steps=3, size_range=((4, 9), (3, 6), (4, 9)))
    with BT.TissueBatch(wl.grids, dt=1 / 60, substeps=3, ks=1e6, stiffness_scale=wl.stiffness_scale(),
                        grasp_params=GraspParams(**dict(W.DEFAULT_GRASP, ccd_velocity=0.0)), dll_path=debug_lib) as b:
        b.set_gravity(0.0, -981.0, 0.0)
        b.set_capsules(wl.capsules_at(0))
        for k in range(3):
            b.step_many([wl.capsules_at(k + 1)], use_graph=k % 2 == 1)
        record = _read(b.dll, "GBT_BatchDebugBoundsRead")
        assert np.isfinite(b.positions()).all()
        assert record[0] == 0, f"{record[0]} out-of-range gathers, first index {record[1]} at site {record[2]}"
        assert checks(b.dll, "GBT_BatchDebugBrickChecks") > 0
