"""What the comparisons of bricks with other shapes rest on: in automatic mode (batches: mode 0) the frames,
rollouts and batches of the cases in test_bricks.py and test_batch.py run on bricks, and those that cannot do not."""
import ctypes as ct

import numpy as np
import pytest

from genesis_tissue_simulation_gb300 import batch as BT
from genesis_tissue_simulation_gb300 import diff as DF
from genesis_tissue_simulation_gb300.native_backend import GraspParams, PlainTissue
from test_debug_bounds import _read, debug_lib  # noqa: F401  (fixture)
from test_guard_bricks import GRASP, arm_guard, block, press

pytestmark = pytest.mark.gpu


def ran(dll, name="GBT_FrameBricks", n=1):
    out = (ct.c_int * n)()
    assert getattr(dll, name)(out) == 0
    return list(out)


@pytest.fixture
def brick_count(gpu_lib):
    dll = ct.CDLL(str(gpu_lib))

    def choose(count):
        assert dll.GBT_SetBrickCount(count) == 0
    yield choose
    dll.GBT_SetBrickCount(0)


@pytest.mark.parametrize("bricks", [1, 5, 152])
def test_guard_and_friction_run_on_bricks(gpu_lib, brick_count, bricks):
    from test_friction_contact import friction_run
    from test_guard import guarded_run
    brick_count(bricks)
    seen = []
    for mode in (0, 1):
        guarded_run(gpu_lib, steps=1, launch_mode=mode, on_close=lambda s: seen.append(ran(s.dll)[0]))
        friction_run(gpu_lib, steps=1, closing=True, launch_mode=mode, on_close=lambda s: seen.append(ran(s.dll)[0]))
    assert seen[2:] == [0, 0]
    for count in seen[:2]:
        assert count == 1 if bricks == 1 else 1 < count <= bricks


def test_the_reported_shape_follows_the_frame(gpu_lib):
    with PlainTissue(block((9, 6, 7)), dt=1 / 60, substeps=3, ks=1e6, strain_damping_s=0.0, grasp_params=GraspParams(**GRASP), dll_path=gpu_lib) as t:
        try:
            assert ran(t.dll) == [0]   # no frame yet
            for mode, on in ((0, True), (1, False), (0, True)):
                assert t.dll.LCS_SetLaunchMode(mode) == 0
                press(t, 0)
                t.step()
                assert (ran(t.dll)[0] > 0) == on
            t.set_tet_stiffness(*t.tet_stiffness())
            arm_guard(t, passes=2)   # carries multipliers between passes: not on bricks
            t.step()
            assert ran(t.dll) == [0]
        finally:
            t.dll.LCS_SetLaunchMode(0)


@pytest.mark.parametrize("size,damping,bricks", [((2, 2, 2), 0.0, 1), ((11, 6, 13), 0.0, 0), ((11, 6, 13), 0.04, 7), ((9, 4, 5), 0.04, 30),
                                                 ((32, 8, 16), 0.0, 0)])
def test_rollouts_run_on_bricks(gpu_lib, brick_count, size, damping, bricks):
    import torch
    brick_count(bricks)
    with DF.DifferentiableTissue(block(size), dt=1 / 60, substeps=2, ks=1e6, strain_damping_s=damping, checkpoint_every=3, max_frames=1,
                                 dll_path=gpu_lib) as t:
        x = t.forward(torch.full((t.tet_count,), float(np.log(1e-6)), device="cuda"), None, frames=1)
        assert ran(t.session.dll, "GBT_DiffBricks", 2)[0] > 0
        t.backward(torch.ones_like(x))
        forward, backward = ran(t.session.dll, "GBT_DiffBricks", 2)
        assert forward == backward and (forward == 1) == (bricks == 1)


@pytest.mark.parametrize("count,lo,hi,damping,ks", [(1, 3, 5, 0.0, 1e6), (3, 4, 9, 0.04, 1e6), (5, 4, 12, 0.04, 0.0), (200, 3, 5, 0.0, 1e6)])
def test_batches_run_on_bricks(gpu_lib, count, lo, hi, damping, ks):
    wl = BT.make_c4(count=count, seed=5, steps=1, size_range=((lo, hi), (3, max(4, hi // 2)), (lo, hi)))
    with BT.TissueBatch(wl.grids, dt=1 / 60, substeps=2, ks=ks, strain_damping_s=damping, grasp_params=GraspParams(**GRASP), dll_path=gpu_lib) as b:
        for use_graph in (False, True):
            b.step_many([wl.capsules_at(1)], use_graph=use_graph)
            assert ran(b.dll, "GBT_BatchFrameBricks")[0] >= count
        b.set_launch(1, 256)
        b.step()
        assert ran(b.dll, "GBT_BatchFrameBricks") == [0]


# bends keep the predict of the next substep in the velocity pass, perpendicular damping takes it out
@pytest.mark.parametrize("material", [dict(kb=1e2, cb=1e-3), dict(cs=1e-3)], ids=["bends", "perpendicular"])
def test_lockstep_on_implicit_codes_matches_the_other_shapes(gpu_lib, debug_lib, monkeypatch, material):  # noqa: F811
    """The lockstep grid with implicit element codes, which serves the batches that cannot run on bricks, against the
    same grid with explicit tables, against one CTA an instance, and with its indices checked."""
    plain = BT.GbtBatchParams

    def params(*fields):
        p = plain(*fields)
        for name, value in material.items():
            setattr(p, name, value)
        return p
    monkeypatch.setattr(BT, "GbtBatchParams", params)
    wl = BT.make_c4(count=7, seed=11, steps=4, size_range=((4, 9), (3, 6), (4, 9)))
    runs = []
    for lib, mode, implicit in ((gpu_lib, 0, True), (gpu_lib, 0, False), (gpu_lib, 1, True), (debug_lib, 0, True)):
        with BT.TissueBatch(wl.grids, dt=1 / 60, substeps=4, ks=1e6, stiffness_scale=wl.stiffness_scale(),
                            grasp_params=GraspParams(**GRASP), dll_path=lib) as b:
            b.set_element_tables(implicit)
            assert b.element_tables() == ("implicit" if implicit else "explicit")
            b.set_launch(mode, 256)
            b.set_gravity(0.0, -981.0, 0.0)
            b.set_capsules(wl.capsules_at(0))
            for k in range(4):
                b.step_many([wl.capsules_at(k + 1)], use_graph=k % 2 == 1)
                assert ran(b.dll, "GBT_BatchFrameBricks") == [0]
            runs.append(b.positions())
            assert lib is gpu_lib or _read(b.dll, "GBT_BatchDebugBoundsRead")[0] == 0
    assert np.isfinite(runs[0]).all()
    for other in runs[1:]:
        assert np.array_equal(runs[0], other)
