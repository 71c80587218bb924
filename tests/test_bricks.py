"""Plain frames on spatial bricks: any brick count, lattice shape, damping and option gives the frame
of the whole-GPU kernel bit for bit, and the oracle's."""
import ctypes as ct

import numpy as np
import pytest

from genesis_tissue_simulation_gb300.grid import build_grid
from genesis_tissue_simulation_gb300 import workloads as W
from genesis_tissue_simulation_gb300.native_backend import Capsule, GraspParams, PlainTissue, blade_sweep

pytestmark = pytest.mark.gpu

# 2 x 2 x 2 cells, a column, a sheet, odd blocks; bricks from one to one per few nodes
LATTICES = {(2, 2, 2): (1, 2, 8), (2, 9, 2): (1, 3, 30), (17, 3, 11): (1, 4, 61), (9, 6, 13): (1, 2, 27, 152)}


def frames(lib, size, bricks=0, mode=0, damping=0.0, ks=1e6, capsule=True, steps=3, substeps=5, blade_at=None, crossing=False, tear=0.0):
    grid = build_grid(0.2, size=tuple(np.float64(c) * 0.2 - 0.02 for c in size), density=1000.0)
    dll = ct.CDLL(str(lib))
    gpu = hasattr(dll, "GBT_SetBrickCount")
    if gpu:
        assert dll.GBT_SetBrickCount(bricks) == 0
    with PlainTissue(grid, dt=1 / 60, substeps=substeps, ks=ks, strain_damping_s=damping, tear_ratio=tear, grasp_params=GraspParams(**W.DEFAULT_GRASP),
                     dll_path=lib) as t:   # contact parameters outlive a session
        info = np.zeros(4, np.int32)
        try:
            if gpu:
                assert dll.LCS_SetLaunchMode(mode) == 0
                assert dll.GBT_BrickInfo(info.ctypes.data_as(ct.c_void_p)) == 0
            t.set_gravity(0.0, -981.0, 0.0)
            top = float(grid.positions[grid.active != 0, 1].max())
            mid = grid.positions[grid.active != 0].mean(axis=0)
            for k in range(steps):
                if capsule:
                    t.set_capsule(Capsule((mid[0] - 1.0, top + 0.2 - 0.06 * k, mid[2]), (mid[0] + 1.0, top + 0.2 - 0.06 * k, mid[2]), 0.25))
                detect = blade_at == k
                if detect:
                    t.set_blade(blade_sweep((mid[0], top + 1.0, mid[2] - 0.3), (mid[0], mid[1], mid[2] - 0.3),
                                            (mid[0], top + 1.0, mid[2] + 0.3), (mid[0], mid[1], mid[2] + 0.3)))
                if crossing:   # a blade through the block, a little further every frame
                    z0, z1 = mid[2] - 0.5 + 0.15 * k, mid[2] - 0.35 + 0.15 * k
                    t.set_blade(blade_sweep((mid[0] + 0.02, top + 1.0, z0), (mid[0] + 0.02, mid[1], z0),
                                            (mid[0] + 0.02, top + 1.0, z1), (mid[0] + 0.02, mid[1], z1)))
                t.step(detect_cut=detect or crossing)
                if detect:   # the blade is put away: plain frames of a severed lattice follow
                    t.functions["LCS_SetPressureCutMode"](1)
            rot = np.zeros((len(grid.positions), 9), np.float32)
            t.check("GBT_GetParticleRot", rot.ctypes.data_as(ct.c_void_p))
            return (t.positions(), t.velocities(), t.neighbors(), rot), info
        finally:
            if gpu:
                dll.LCS_SetLaunchMode(0)
                dll.GBT_SetBrickCount(0)


@pytest.mark.parametrize("size,bricks", [(s, b) for s, counts in LATTICES.items() for b in counts])
@pytest.mark.parametrize("options", [dict(), dict(damping=0.04), dict(damping=0.04, ks=0.0), dict(ks=0.0, capsule=False)],
                         ids=["plain", "damped", "damped-fallback", "fallback"])
def test_bricks_match_the_whole_gpu_frame(gpu_lib, size, bricks, options):
    got, info = frames(gpu_lib, size, bricks, **options)
    want, _ = frames(gpu_lib, size, mode=1, **options)
    assert info[0] >= 1 and (bricks == 1) == (info[0] == 1)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("bricks", [1, 5, 40])
def test_bricks_match_the_oracle_through_a_cut(gpu_lib, oracle_libs, bricks):
    """Frames before and after a blade frame: the live bits follow the severed links."""
    got, _ = frames(gpu_lib, (9, 6, 13), bricks, steps=6, blade_at=2)
    want, _ = frames(oracle_libs[0], (9, 6, 13), steps=6, blade_at=2)
    assert (got[2] != want[2]).sum() == 0 and (got[2] < 0).sum() > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("size,bricks", [((9, 6, 13), 1), ((9, 6, 13), 27), ((17, 3, 11), 61)])
@pytest.mark.parametrize("options", [dict(), dict(damping=0.04), dict(tear=1.05)], ids=["plain", "damped", "tear"])
def test_blade_frames_on_bricks_match_the_whole_gpu_frame(gpu_lib, size, bricks, options):
    """Ticks between the substeps of frames whose links the rod-phase detection severs, and the particle frames after them."""
    got, info = frames(gpu_lib, size, bricks, steps=6, crossing=True, **options)
    want, _ = frames(gpu_lib, size, mode=1, steps=6, crossing=True, **options)
    start = build_grid(0.2, size=tuple(np.float64(c) * 0.2 - 0.02 for c in size), density=1000.0).neighbors
    assert info[0] >= 1 and (want[2] != start).sum() > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_a_lost_neighbour_ends_the_frame_with_a_status(gpu_lib):
    """Exchanges that await an epoch nobody publishes give up within the budget; the next frame is sound."""
    dll = ct.CDLL(str(gpu_lib))
    dll.LCS_SetBarrierTest.argtypes = (ct.c_int, ct.c_float)
    grid = build_grid(0.2, size=(1.78, 1.18, 2.58), density=1000.0)
    assert dll.GBT_SetBrickCount(8) == 0
    try:
        with PlainTissue(grid, dt=1 / 60, substeps=2, ks=1e6, strain_damping_s=0.0, dll_path=gpu_lib) as t:
            assert dll.LCS_SetBarrierTest(1, 0.05) == 0
            with pytest.raises(RuntimeError, match="-4002"):
                t.step()
            assert dll.LCS_SetBarrierTest(0, 2.0) == 0
            t.step()
    finally:
        dll.LCS_SetBarrierTest(0, 2.0)
        dll.GBT_SetBrickCount(0)


@pytest.mark.parametrize("size,damping,bricks", [((2, 2, 2), 0.0, 1), ((11, 6, 13), 0.0, 0), ((11, 6, 13), 0.04, 7), ((9, 4, 5), 0.04, 30),
                                                 ((32, 8, 16), 0.0, 0)])
def test_rollouts_on_bricks_match_the_whole_gpu_rollout(gpu_lib, size, damping, bricks):
    """Forward bit for bit; adjoints to the rounding of signed-zero terms and of the path sum's order."""
    import torch

    from genesis_tissue_simulation_gb300 import diff as D
    grid = build_grid(0.2, size=tuple(np.float64(c) * 0.2 - 0.02 for c in size), density=1000.0)
    top = float(grid.positions[grid.active != 0, 1].max())
    mid = grid.positions[grid.active != 0].mean(axis=0)
    path = np.array([[mid[0] - 0.5, top + 0.2 - 0.1 * k, mid[2], mid[0] + 0.5, top + 0.2 - 0.1 * k, mid[2]] for k in range(4)], np.float32)
    dll = ct.CDLL(str(gpu_lib))
    out = []
    for mode in (0, 1):
        assert dll.GBT_SetBrickCount(bricks) == 0
        try:
            with D.DifferentiableTissue(grid, dt=1 / 60, substeps=4, ks=1e6, strain_damping_s=damping, gravity=(0.0, -981.0, 0.0),
                                        checkpoint_every=3, max_frames=3, launch_mode=mode, dll_path=gpu_lib, scale_modulus=1e6) as t:
                rng = np.random.default_rng(3)
                theta = torch.tensor(np.log(1e-6) + rng.uniform(-0.5, 0.5, t.tet_count), dtype=torch.float32, device="cuda")
                g = torch.tensor(rng.standard_normal((t.n_nodes, 3)), dtype=torch.float32, device="cuda")
                for _ in range(2):   # a second rollout on the same handle starts from the same origin
                    x = t.forward(theta, torch.tensor(path, device="cuda"))
                    adj = t.backward(g, rest_shape=True, origin=True)
                out.append((x.cpu().numpy(), {k: v.cpu().numpy() for k, v in adj.items()}, t.session.velocities(), t.info()))
        finally:
            dll.GBT_SetBrickCount(0)
            dll.LCS_SetLaunchMode(0)
    (x, adj, v, info), (x1, adj1, v1, _) = out
    assert bricks == 0 or info["ctas"] == (1 if bricks == 1 else info["ctas"]) and (bricks == 1 or info["ctas"] > 1)
    assert np.array_equal(x, x1) and np.array_equal(v, v1)
    for name, a in adj.items():
        b = adj1[name]
        assert np.isfinite(a).all()
        # path: 12 substeps' sums in another order; the rest differs at most by zeros that were added
        assert np.abs(a - b).max() <= (1e-5 if name == "path" else 1e-6) * max(np.abs(b).max(), 1e-30), name


@pytest.mark.parametrize("bricks", [1, 5, 152])
@pytest.mark.parametrize("minimum", [0.15, 0.9])
def test_guarded_frames_on_bricks_match_the_whole_gpu_frame(gpu_lib, bricks, minimum):
    """The guard's tet form, its tensile pass and its feasibility chain (which 0.9 sets off)."""
    from test_guard import guarded_run
    dll = ct.CDLL(str(gpu_lib))
    assert dll.GBT_SetBrickCount(bricks) == 0
    try:
        _, got, _ = guarded_run(gpu_lib, steps=6, minimum=minimum, launch_mode=0)
    finally:
        dll.GBT_SetBrickCount(0)
    _, want, _ = guarded_run(gpu_lib, steps=6, minimum=minimum, launch_mode=1)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("bricks", [1, 5, 152])
def test_friction_frames_on_bricks_match_the_whole_gpu_frame(gpu_lib, bricks):
    from test_friction_contact import friction_run
    dll = ct.CDLL(str(gpu_lib))
    assert dll.GBT_SetBrickCount(bricks) == 0
    try:
        _, got = friction_run(gpu_lib, steps=6, closing=True, launch_mode=0)
    finally:
        dll.GBT_SetBrickCount(0)
    _, want = friction_run(gpu_lib, steps=6, closing=True, launch_mode=1)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
