"""Performance cases of the tissue solver, through its public entry points.

Five kinds of pass, over the ranges a simulator, a viewer or an identification loop uses:

* ``step``: one frame of a single session (command, ``PlainTissue.step``, node state out), from the
  600-voxel block of the adapter's default grid to the 64 x 32 x 48 kidney-scale block; with the
  adapter's settings (no lattice edges stiffness, strain damping), a pressed capsule, or the tissue
  guard with a grasping jaw pair;
* ``view``: the same frame plus the reconstructed surface, what a viewer draws;
* ``cut``: a blade frame with rod-phase detection, then the cut mesh re-coloured as an unstructured
  tet mesh;
* ``batch``: frames of many uneven instances in one launch, replayed from a CUDA graph;
* ``rollout``: the differentiable rollout, forward alone or with its adjoint.

The library serves one session per loaded plugin, so every state loads its own copy of it (a small
pool, one copy per live state), as a program with several environments in one process does.
"""
import ctypes as ct
import math
import shutil
import tempfile
from pathlib import Path

import numpy as np
import torch

from genesis_tissue_simulation_gb300 import batch as BT
from genesis_tissue_simulation_gb300 import diff as DF
from genesis_tissue_simulation_gb300 import workloads as W
from genesis_tissue_simulation_gb300.grid import METERS_PER_UNIT, build_grid
from genesis_tissue_simulation_gb300.native_backend import (DEFAULT_DLL, Capsule, Grasper, GraspParams, PlainTissue, V3,
                                                            blade_sweep, pointer)

DT = 1 / 60
YOUNG, POISSON, SPACING = 6000.0, 0.25, 0.2
GRAVITY = (0.0, -981.0, 0.0)
GRASP = dict(W.DEFAULT_GRASP, ccd_velocity=0.0)
# seconds of double-precision work beyond which exact() gives no value (vector operations per colour)
EXACT_LIMIT_TETS = 7e6


# -------------------------------------------------------------------------------------------------
# cases
# -------------------------------------------------------------------------------------------------
def listed():
    return [
        # the adapter's default block (6 mm voxels, 352 active nodes) with the adapter's frame (1/30 s,
        # 3 substeps, strain damping, no edge stiffness): an interactive loop at its smallest
        {"name": "adapter_block", "kind": "step", "spacing": 0.6, "x": 0, "y": 0, "z": 0, "substeps": 3, "ks": 0.0, "damping": 0.04,
         "tool": "none"},
        # the plain 16 x 8 x 16 block, 10 substeps
        {"name": "plain_16x8x16", "kind": "step", "spacing": SPACING, "x": 16, "y": 8, "z": 16, "substeps": 10, "ks": 1e6,
         "damping": 0.0, "tool": "none"},
        # an ordinary session of odd size with a capsule pressed in and out of its top
        {"name": "capsule_23x13x19", "kind": "step", "spacing": SPACING, "x": 23, "y": 13, "z": 19, "substeps": 20, "ks": 1e6,
         "damping": 0.0, "tool": "capsule"},
        # the kidney-scale block with the capsule, 20 substeps: the headline workload
        {"name": "capsule_64x32x48", "kind": "step", "spacing": SPACING, "x": 64, "y": 32, "z": 48, "substeps": 20, "ks": 1e6,
         "damping": 0.0, "tool": "capsule"},
        # tissue guard and a jaw pair with friction: the options of a grasping session
        {"name": "guarded_jaws_16x8x16", "kind": "step", "spacing": SPACING, "x": 16, "y": 8, "z": 16, "substeps": 10, "ks": 1e6,
         "damping": 0.04, "tool": "jaws"},
        # a viewer: a frame, its surface triangles and the nodes
        {"name": "view_30x12x22", "kind": "view", "spacing": SPACING, "x": 30, "y": 12, "z": 22, "substeps": 10, "ks": 1e6,
         "damping": 0.0, "tool": "capsule"},
        # the kidney-scale block under the blade, re-coloured after every frame
        {"name": "blade_64x32x48", "kind": "cut", "x": 64, "y": 32, "z": 48, "substeps": 20},
        # a handful of small uneven instances, 4 frames a call
        {"name": "batch_12", "kind": "batch", "count": 12, "sizes": 4, "lo": 8, "hi": 20, "frames": 4, "substeps": 10},
        # 256 uneven instances (8..32 x 4..16 x 8..32 cells), 2 frames a call
        {"name": "batch_256", "kind": "batch", "count": 256, "sizes": 4, "lo": 8, "hi": 32, "frames": 2, "substeps": 10},
        # forward rollouts alone: evaluating a material estimate on the 32 x 16 x 32 block
        {"name": "rollout_32x16x32", "kind": "rollout", "x": 32, "y": 16, "z": 32, "frames": 20, "substeps": 10, "grad": False},
        # one identification step on the same block: forward, loss, adjoint
        {"name": "identify_32x16x32", "kind": "rollout", "x": 32, "y": 16, "z": 32, "frames": 20, "substeps": 10, "grad": True},
        # the same on a small odd block
        {"name": "identify_11x6x13", "kind": "rollout", "x": 11, "y": 6, "z": 13, "frames": 4, "substeps": 10, "grad": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "view", "cut", "batch", "batch", "rollout", "rollout"])
    x, y, z = _log(rng, 3, 64), _log(rng, 3, 32), _log(rng, 3, 48)
    if kind in ("step", "view"):
        tool = rng.choice(["none", "capsule", "capsule", "jaws"]) if kind == "step" else rng.choice(["none", "capsule"])
        damped = tool == "jaws" or rng.random() < 0.2
        if tool == "jaws":
            x, y, z = min(x, 24), min(y, 12), min(z, 24)
        if damped:
            y = min(y, 8)   # strain damping at these substep lengths flattens taller blocks
        return {"kind": kind, "spacing": SPACING, "x": x, "y": y, "z": z, "substeps": rng.randint(3, 20),
                "ks": 0.0 if damped and tool == "none" and rng.random() < 0.5 else 1e6, "damping": 0.04 if damped else 0.0,
                "tool": tool}
    if kind == "cut":
        return {"kind": kind, "x": max(x, 8), "y": max(y, 4), "z": max(z, 8), "substeps": rng.randint(3, 20)}
    if kind == "batch":
        lo = rng.randint(4, 10)
        return {"kind": kind, "count": _log(rng, 2, 128), "sizes": rng.randrange(1 << 16), "lo": lo, "hi": rng.randint(lo + 2, 32),
                "frames": rng.randint(1, 4), "substeps": rng.randint(4, 10)}
    return {"kind": kind, "x": _log(rng, 4, 32), "y": _log(rng, 3, 16), "z": _log(rng, 4, 32), "frames": rng.randint(1, 12),
            "substeps": rng.randint(4, 10), "grad": rng.random() < 0.6}


# -------------------------------------------------------------------------------------------------
# what a program has in hand
# -------------------------------------------------------------------------------------------------
class _Plugins:
    """Paths of library copies; a closed state's copy is given back."""
    folder = None
    free = []
    made = 0

    @classmethod
    def take(cls):
        if cls.free:
            return cls.free.pop()
        if cls.folder is None:
            cls.folder = tempfile.TemporaryDirectory(prefix="tissue_plugins_")
        path = Path(cls.folder.name) / f"plugin{cls.made}.so"
        cls.made += 1
        shutil.copyfile(DEFAULT_DLL, path)
        return path


class _State:
    """A session (or batch) on its own copy of the library, its inputs and its command counter."""

    def __init__(self, case):
        self.case, self.path, self.handle, self.k = case, _Plugins.take(), None, 0

    def __del__(self):
        if self.handle is not None:
            self.handle.close()
        _Plugins.free.append(self.path)


_GRIDS = {}


def _grid(spacing, x, y, z):
    """The block of x, y (up), z cells; x = 0: the adapter's default block."""
    key = (spacing, x, y, z)
    if key not in _GRIDS:
        _GRIDS[key] = build_grid(spacing) if x == 0 else build_grid(spacing, size=tuple(np.float64(c) * spacing - 0.02 for c in (x, y, z)),
                                                                    density=1000.0)
    return _GRIDS[key]


def _full_cells(grid):
    a = (grid.active != 0).reshape(grid.dims[2] + 1, grid.dims[1] + 1, grid.dims[0] + 1)
    return (a[:-1, :-1, :-1] & a[1:, :-1, :-1] & a[:-1, 1:, :-1] & a[1:, 1:, :-1] & a[:-1, :-1, 1:] & a[1:, :-1, 1:]
            & a[:-1, 1:, 1:] & a[1:, 1:, 1:])


def _tets(grid):
    return 6 * int(_full_cells(grid).sum())


def _volume(grid):
    return np.float32(float(np.prod(np.asarray(grid.cell_size, dtype=np.float64))) / 6.0)


def _stiffness(grid, seed):
    """(mu V, kappa V) per tet: a seeded compliance per tet, log-uniform in [1e-7, 1e-5] 1/Pa."""
    rng = np.random.default_rng(seed)
    n = _tets(grid)
    young = 1.0 / np.exp(rng.uniform(math.log(1e-7), math.log(1e-5), n)) * METERS_PER_UNIT
    v = float(_volume(grid))
    return ((young / (2 * (1 + POISSON))) * v).astype(np.float32), ((young / (3 * (1 - 2 * POISSON))) * v).astype(np.float32)


def _state_of(grid, seed):
    """Node positions and velocities of a running session: the rest lattice under a smooth seeded
    displacement (0.02 cm) and a smooth velocity field (0.5 cm/s); the pinned bed at rest."""
    rng = np.random.default_rng(seed + 1)
    p = grid.positions.astype(np.float64)
    free = ((grid.active != 0) & (grid.pinned == 0))[:, None]
    rise = np.clip((p[:, 1:2] - p[grid.active != 0, 1].min()) / 2.0, 0.0, 1.0)
    k = rng.uniform(-1.0, 1.0, (2, 3, 3))
    phase = rng.uniform(0, 2 * np.pi, (2, 3))
    u = np.stack([np.sin(p @ k[0, a] + phase[0, a]) for a in range(3)], axis=1)
    v = np.stack([np.sin(p @ k[1, a] + phase[1, a]) for a in range(3)], axis=1)
    pos = np.where(free, p + 0.02 * rise * u, p).astype(np.float32)
    vel = np.where(free, 0.5 * rise * v, 0.0).astype(np.float32)
    return np.ascontiguousarray(pos), np.ascontiguousarray(vel)


def _extent(grid):
    p = grid.positions[grid.active != 0]
    return p.min(axis=0).astype(np.float64), p.max(axis=0).astype(np.float64)


def _capsules(grid, seed, steps):
    """Capsule poses [steps + 1, 7]: pressed from just inside the top to 0.6 cm (or a third of the
    height), then withdrawn, over ``steps`` frames."""
    rng = np.random.default_rng(seed + 2)
    lo, hi = _extent(grid)
    mid, half = (lo + hi) / 2, (hi - lo) / 2
    angle = rng.uniform(0.0, np.pi)
    axis = np.array((np.cos(angle), 0.0, np.sin(angle)))
    r, length = 0.25, min(4.0, 1.2 * min(half[0], half[2]))
    c = mid + np.array((rng.uniform(-0.3, 0.3) * half[0], 0.0, rng.uniform(-0.3, 0.3) * half[2]))
    depth = min(0.6, (hi[1] - lo[1]) / 3)
    out = np.zeros((steps + 1, 7), dtype=np.float32)
    for k in range(steps + 1):
        f = 2.0 * k / steps if 2 * k <= steps else 2.0 - 2.0 * k / steps
        at = np.array((c[0], hi[1] + r - 0.02 - depth * f, c[2]))
        out[k] = (*(at - axis * length / 2), *(at + axis * length / 2), r)
    return out


def _capsule(row):
    return Capsule(tuple(float(v) for v in row[:3]), tuple(float(v) for v in row[3:6]), float(row[6]))


def _jaws(grid, seed, steps):
    """A jaw pair closing on the top face and opening again."""
    rng = np.random.default_rng(seed + 3)
    lo, hi = _extent(grid)
    mid = (lo + hi) / 2
    x, z = mid[0] + rng.uniform(-0.3, 0.3), mid[2] + rng.uniform(-0.3, 0.3)
    poses = []
    for k in range(steps + 1):
        f = 2.0 * k / steps if 2 * k <= steps else 2.0 - 2.0 * k / steps
        y, gap = hi[1] + 0.45 - 0.5 * f, 0.5 - 0.3 * f
        poses.append(Grasper(V3(x - 0.4, y + 0.9, z), V3(x + 0.4, y + 1.6, z), 0.25, V3(x - 0.6, y, z), V3(1.0, 0.0, 0.15), V3(x, y, z),
                             V3(0.0, 1.0, 0.0), 0.35, 1.2, gap, 0.0))
    return poses


def _blade(grid, seed, lane):
    """Blade sweeps of one crossing in x, 200 frames along a seeded polyline, its lower edge 1 cm (or
    half the height) below the top; each lane lies beside the one before."""
    rng = np.random.default_rng(seed + 4)
    lo, hi = _extent(grid)
    mid, half = (lo + hi) / 2, (hi - lo) / 2
    xs = mid[0] + np.linspace(-0.8 * half[0], 0.8 * half[0], 13)
    zs = mid[2] + np.clip(np.cumsum(rng.uniform(-0.35, 0.35, 13)) * half[2] * 0.3, -0.35 * half[2], 0.35 * half[2])
    zs = zs + ((lane * 0.618034 + 0.5) % 1.0 - 0.5) * half[2]
    y0 = hi[1] - min(1.0, (hi[1] - lo[1]) / 2)
    s = np.linspace(0, 12, 201)
    px, pz = np.interp(s, np.arange(13), xs), np.interp(s, np.arange(13), zs)
    ends = [((px[k], y0 + 3.0, pz[k]), (px[k], y0, pz[k])) for k in range(201)]
    return [blade_sweep(*ends[k], *ends[k + 1]) for k in range(200)]


def _set_state(session, pos, vel):
    f = session.dll.GBT_SetState
    f.argtypes, f.restype = (ct.c_void_p,) * 8 + (ct.c_int32, ct.c_uint32), ct.c_int32
    rc = f(pointer(pos), pointer(vel), *([None] * 6), 0, 0)
    if rc != 0:
        raise RuntimeError(f"GBT_SetState failed with native status {rc}")


PRESS = 60   # frames of one press and withdrawal


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    if kind in ("step", "view", "cut"):
        grid = _grid(case.get("spacing", SPACING), case["x"], case["y"], case["z"])
        mu, kappa = (None, None) if case["x"] == 0 else _stiffness(grid, seed)
        if case.get("tool") == "jaws":   # contact model 1 meets the nodes of a lattice without a surface
            grid = type(grid)(**{**vars(grid), "surface_edges": np.zeros((0, 8), dtype=np.int32)})
        dt = 1 / 30 if case["x"] == 0 else DT
        s.handle = t = PlainTissue(grid, dt=dt, substeps=case["substeps"], ks=case.get("ks", 1e6), young_pa=YOUNG, poisson=POISSON,
                                   strain_damping_s=case.get("damping", 0.0), tet_mu_v=mu, tet_kappa_v=kappa,
                                   grasp_params=GraspParams(**GRASP), dll_path=s.path)
        t.set_gravity(*GRAVITY)
        if case.get("tool") == "jaws":
            t.check("LCS_SetTissueGuard", ct.c_float(0.15), 1, len(grid.positions), pointer(grid.inside), 1)
            t.check("LCS_SetContactModel", 1, ct.c_float(0.6), ct.c_float(0.4), ct.c_float(0.1), ct.c_float(0.01))
            s.commands = _jaws(grid, seed, PRESS)
            t.check("LCS_SetGraspTool", ct.byref(s.commands[0]))
        elif case.get("tool") == "capsule":
            s.commands = [_capsule(r) for r in _capsules(grid, seed, PRESS)]
            t.set_capsule(s.commands[0])
        elif kind == "cut":
            s.grid, s.seed, s.lane, s.commands = grid, seed, 0, _blade(grid, seed, 0)
        _set_state(t, *_state_of(grid, seed))
    elif kind == "batch":
        grids = _instances(case)
        rng = np.random.default_rng(seed)
        compliance = np.exp(rng.uniform(math.log(1e-7), math.log(1e-5), len(grids)))
        scale = (1.0 / (compliance * YOUNG)).astype(np.float32)
        s.handle = b = BT.TissueBatch(grids, dt=DT, substeps=case["substeps"], ks=1e6, young_pa=YOUNG, poisson=POISSON,
                                      strain_damping_s=0.0, stiffness_scale=scale, grasp_params=GraspParams(**GRASP), dll_path=s.path)
        b.set_gravity(*GRAVITY)
        s.commands = np.stack([_capsules(g, seed + i, PRESS) for i, g in enumerate(grids)], axis=1)
        b.set_capsules([_capsule(r) for r in s.commands[0]])
        if case["count"] <= 64:   # a large table keeps the default launch, which is what the tuner keeps there
            b.autotune(2)
        s.out = np.empty((b.total_nodes, 3), dtype=np.float32)
    else:
        grid = _grid(SPACING, case["x"], case["y"], case["z"])
        s.handle = DF.DifferentiableTissue(grid, dt=DT, substeps=case["substeps"], ks=1e6, young_pa=YOUNG, poisson=POISSON,
                                           strain_damping_s=0.0, gravity=GRAVITY, grasp_params=GraspParams(**GRASP),
                                           checkpoint_every=5, max_frames=case["frames"], dll_path=s.path, scale_modulus=1e6)
        theta, path, target = _material(case, grid, seed)
        s.theta = torch.tensor(theta, device="cuda", requires_grad=case["grad"])
        s.route = torch.tensor(path, device="cuda", requires_grad=case["grad"])
        s.target = torch.tensor(target, device="cuda")
        top = float(grid.positions[grid.active != 0, 1].max())
        s.top = torch.tensor(np.nonzero((grid.active != 0) & (np.abs(grid.positions[:, 1] - top) < 1e-6))[0], device="cuda")
    return s


def _material(case, grid, seed):
    """Per-tet log-compliance around 1e-6 1/Pa, the capsule route of the rollout, and target positions
    of the nodes: the rest lattice under a smooth dent."""
    rng = np.random.default_rng(seed)
    theta = (math.log(1e-6) + rng.uniform(-0.5, 0.5, _tets(grid))).astype(np.float32)
    path = _capsules(grid, seed, 2 * case["frames"])[:case["frames"] + 1, :6]
    target, _ = _state_of(grid, seed)
    return theta, np.ascontiguousarray(path), target


def _instances(case):
    rng = np.random.default_rng(case["sizes"])
    lo, hi = case["lo"], case["hi"]
    return [_grid(SPACING, int(rng.integers(lo, hi + 1)), int(rng.integers(max(lo // 2, 3), hi // 2 + 1)), int(rng.integers(lo, hi + 1)))
            for _ in range(case["count"])]


# -------------------------------------------------------------------------------------------------
# one pass
# -------------------------------------------------------------------------------------------------
def run(state):
    case, kind = state.case, state.case["kind"]
    if kind in ("step", "view"):
        t = state.handle
        if case["tool"] != "none":
            state.k = state.k % PRESS + 1
            if case["tool"] == "capsule":
                t.set_capsule(state.commands[state.k])
            else:
                t.check("LCS_SetGraspTool", ct.byref(state.commands[state.k]))
        t.step()
        if kind == "view":
            surface = t.surface()
            return [t.positions(), surface["pos"], surface["nrm"], surface["tri"]]
        return [t.positions(), t.velocities()]
    if kind == "cut":
        t = state.handle
        if state.k == len(state.commands):
            state.k, state.lane = 0, state.lane + 1
            state.commands = _blade(state.grid, state.seed, state.lane)
        t.set_blade(state.commands[state.k])
        state.k += 1
        t.step(detect_cut=True)
        mesh = t.cut_topology()
        return [t.positions(), t.neighbors(), mesh["tet_nodes"], mesh["tet_colour"], mesh["dup_parent"]]
    if kind == "batch":
        at = [(state.k + j) % PRESS + 1 for j in range(case["frames"])]
        state.k = at[-1]
        state.handle.step_many(np.ascontiguousarray(state.commands[at]))
        return [state.handle.positions(out=state.out)]
    if not case["grad"]:
        return [state.handle.rollout(state.theta, state.route)]
    state.theta.grad = state.route.grad = None
    x = state.handle.rollout(state.theta, state.route)
    DF.identification_loss(x, state.target, state.top).backward()
    return [x.detach(), state.theta.grad, state.route.grad]


# -------------------------------------------------------------------------------------------------
# what a pass cannot do without
# -------------------------------------------------------------------------------------------------
def _counts(grid):
    return int((grid.active != 0).sum()), _tets(grid), int((grid.neighbors[:, 1::2] >= 0).sum())


# floating operations of one projection (a fused multiply-add is two): tet, lattice edge, node pass
TET, EDGE, NODE = 560.0, 45.0, 30.0


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n, t, e = (sum(c) for c in zip(*(_counts(g) for g in _instances(case))))
        frames, nodes = case["frames"], sum(len(g.positions) for g in _instances(case))
    else:
        grid = _grid(case.get("spacing", SPACING), case["x"], case["y"], case["z"])
        n, t, e = _counts(grid)
        frames, nodes = case.get("frames", 1), len(grid.positions)
    edges = e if case.get("ks", 1e6) > 0 else 0
    flops = frames * case["substeps"] * (TET * t + EDGE * edges + NODE * n)
    # positions and velocities in and out, one compliance per tet, the nodes handed to the caller
    moved = 48.0 * n + 4.0 * t + 12.0 * nodes
    if kind == "step":
        moved += 12.0 * nodes
    elif kind == "cut":   # the neighbour table and the cut mesh: four nodes and a colour per tet
        moved += 24.0 * nodes + 20.0 * t
    elif kind == "view":  # about two triangles per surface cell: position, normal and tag per corner
        moved += 84.0 * 2 * 2 * (case["x"] * case["y"] + case["y"] * case["z"] + case["x"] * case["z"])
    elif kind == "rollout":
        saved = frames * case["substeps"] / 5 * 24.0 * n   # the state at every checkpoint
        moved += saved
        if case["grad"]:   # recompute and reverse sweep; checkpoints read, gradients written
            flops *= 4.0
            moved += saved + 16.0 * t + 24.0 * n
    return {"bytes": moved, "flops": flops}


# -------------------------------------------------------------------------------------------------
# the same in double precision
# -------------------------------------------------------------------------------------------------
KUHN = ((0, 1, 3, 7), (0, 3, 2, 7), (0, 2, 6, 7), (0, 6, 4, 7), (0, 4, 5, 7), (0, 5, 1, 7))
_MESHES = {}


def _first_fit(elements, nodes):
    """Greedy colours: each element takes the lowest colour none of its nodes carries yet."""
    taken, colour = [0] * nodes, np.empty(len(elements), dtype=np.int64)
    for i, el in enumerate(elements.tolist()):
        busy = 0
        for n in el:
            busy |= taken[n]
        bit = ~busy & (busy + 1)
        colour[i] = bit.bit_length() - 1
        for n in el:
            taken[n] |= bit
    return colour


def _mesh(spacing, x, y, z):
    """Colour lists of the block's lattice edges and Kuhn tets, rest inverses and storage order."""
    key = (spacing, x, y, z)
    if key in _MESHES:
        return _MESHES[key]
    grid = _grid(*key)
    n = len(grid.positions)
    p, a = np.nonzero(grid.neighbors[:, 1::2] >= 0)
    ends = np.stack((p, grid.neighbors[p, 2 * a + 1]), axis=1).astype(np.int64)
    rest = np.linalg.norm(grid.rest_neighbors.reshape(n, 6, 3)[p, 2 * a + 1].astype(np.float64), axis=1)
    nx, ny = grid.dims[0] + 1, grid.dims[1] + 1
    cz, cy, cx = np.nonzero(_full_cells(grid))
    base = cx + nx * (cy + ny * cz)
    step = np.array([(c & 1) + nx * ((c >> 1 & 1) + ny * (c >> 2 & 1)) for c in range(8)])
    tets = (base[:, None, None] + step[np.array(KUHN)][None]).reshape(-1, 4).astype(np.int64)
    kind = np.tile(np.arange(6), len(base))
    storage = kind * len(base) + np.repeat(np.arange(len(base)), 6)
    cell = [(float(grid.positions[-1, q]) - float(grid.positions[0, q])) / grid.dims[q] for q in range(3)]
    corner = np.array([[c >> q & 1 for q in range(3)] for c in range(8)]) * np.array(cell)
    inverse = np.stack([np.linalg.inv((corner[list(k[1:])] - corner[0]).T) for k in KUHN])
    dev = dict(device="cuda")
    group = lambda colours: [torch.tensor(np.nonzero(colours == c)[0], **dev) for c in range(int(colours.max()) + 1)]  # noqa: E731
    w = np.where((grid.active != 0) & (grid.pinned == 0), 1.0 / np.where(grid.mass > 0, grid.mass.astype(np.float64), 1.0), 0.0)
    m = dict(n=n, ends=torch.tensor(ends, **dev), rest=torch.tensor(rest, **dev), edges=group(_first_fit(ends, n)),
             tets=torch.tensor(tets, **dev), kind=torch.tensor(kind, **dev), storage=torch.tensor(storage, **dev),
             colours=group(_first_fit(tets, n)), inverse=torch.tensor(inverse, **dev), w=torch.tensor(w, **dev),
             mass=torch.tensor(grid.mass.astype(np.float64), **dev), volume=float(np.prod(cell)) / 6.0)
    _MESHES.clear()
    _MESHES[key] = m
    return m


def _substep(m, x, v, mu, kappa, h, ks, damping, capsule):
    """One substep in 64 bits: predict, edge colours, tet colours, capsule contact, velocity."""
    w, free = m["w"], (m["w"] > 0)[:, None]
    q = x
    acc = torch.tensor(GRAVITY, device="cuda", dtype=torch.float64)
    v = torch.where(free, v + acc * h, v)
    x = torch.where(free, x + v * h, x)
    if ks > 0:
        alpha = 1.0 / (ks * h * h)
        for e in m["edges"]:
            i, j = m["ends"][e, 0], m["ends"][e, 1]
            wi, wj = w[i], w[j]
            d = x[i] - x[j]
            length = d.norm(dim=1)
            dl = torch.where(wi + wj > 0, (m["rest"][e] - length) / (wi + wj + alpha), torch.zeros_like(length))
            move = d * (dl / length)[:, None]
            x = x.index_add(0, i, move * wi[:, None]).index_add(0, j, -move * wj[:, None])
    over = damping / h
    for t in m["colours"]:
        ids, st = m["tets"][t], m["storage"][t]
        B = m["inverse"][m["kind"][t]]
        p, wt = x[ids], w[ids]
        F = torch.einsum("tki,tkc->tci", p[:, 1:] - p[:, :1], B)              # column c of F
        cof = torch.stack([torch.linalg.cross(F[:, (c + 1) % 3], F[:, (c + 2) % 3]) for c in range(3)], dim=1)
        I1, J = (F * F).sum((1, 2)), (F[:, 0] * cof[:, 0]).sum(1)
        low = torch.clamp(J, min=0.05)
        iso = low ** (-2.0 / 3.0)
        CD = torch.sqrt(torch.clamp(iso * I1 - 3.0, min=1e-12))
        vol = torch.where(J > 0.05, iso * I1 / (3.0 * low), torch.zeros_like(J))
        gh = torch.einsum("tcj,tji->tci", B, cof)
        gd = (torch.einsum("tcj,tji->tci", B, F) * iso[:, None, None] - gh * vol[:, None, None]) / CD[:, None, None]
        gh = torch.cat((-gh.sum(1, keepdim=True), gh), 1)
        gd = torch.cat((-gd.sum(1, keepdim=True), gd), 1)
        dx = p - q[ids]
        aD, aH = 1.0 / (h * h * mu[st] * (1 + over)), 1.0 / (h * h * kappa[st] * (1 + over))
        A = (wt * (gd * gd).sum(2)).sum(1) + aD
        cross = (wt * (gd * gh).sum(2)).sum(1)
        g = cross / A
        S = aH + aD * g * g + (wt * ((gh - gd * g[:, None, None]) ** 2).sum(2)).sum(1)
        rd = (-CD - over * (gd * dx).sum((1, 2))) / (1 + over)
        rh = (1.0 - J - over * (gh * dx).sum((1, 2))) / (1 + over)
        lh = (rh - g * rd) / S
        ld = (rd - cross * lh) / A
        move = (gd * ld[:, None, None] + gh * lh[:, None, None]) * wt[:, :, None]
        x = x.index_add(0, ids.reshape(-1), move.reshape(-1, 3))
    if capsule is not None:
        a, b, r = capsule
        ab = b - a
        f = torch.clamp(((x - a) * ab).sum(1) / (ab * ab).sum(), 0.0, 1.0)
        d = x - (a + ab * f[:, None])
        dist = d.norm(dim=1)
        safe = torch.where(dist > 1e-9, dist, torch.ones_like(dist))
        nrm = d / safe[:, None]
        hit = (w > 0) & (dist < r) & (-(v * nrm).sum(1) > GRASP["ccd_velocity"])
        push = GRASP["ccd_omega"] * w * (r - dist) / (w + GRASP["contact_compliance"] / (h * h))
        push = torch.clamp(push, max=GRASP["ccd_displacement"])
        x = torch.where(hit[:, None], x + nrm * push[:, None], x)
    return x, torch.where(free, (x - q) / h, torch.zeros_like(x))


def _frame(m, x, v, mu, kappa, dt, substeps, ks, damping, poses):
    h = float(np.float32(dt)) / substeps
    for s in range(substeps):
        f = min(1.0, (s + 1) / substeps)
        capsule = None if poses is None else (poses[0][:3] * (1 - f) + poses[1][:3] * f, poses[0][3:6] * (1 - f) + poses[1][3:6] * f,
                                              0.25)
        x, v = _substep(m, x, v, mu, kappa, h, ks, damping, capsule)
    return x, v


def _wide(a):
    return torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cut", "batch") and (kind == "cut" or case["count"] > 16):
        return None
    if case.get("tool") == "jaws":
        return None
    if kind == "batch":
        grids = _instances(case)
        if case["frames"] * case["substeps"] * sum(_tets(g) for g in grids) > 4 * EXACT_LIMIT_TETS:
            return None
        rng = np.random.default_rng(seed)
        compliance = np.exp(rng.uniform(math.log(1e-7), math.log(1e-5), len(grids)))
        scale = (1.0 / (compliance * YOUNG)).astype(np.float32).astype(np.float64)
        out, e = [], YOUNG * METERS_PER_UNIT
        for i, g in enumerate(grids):
            key = next(k for k, v in _GRIDS.items() if v is g)
            m = _mesh(*key)
            t = m["tets"].shape[0]
            mu = torch.full((t,), e / (2 * (1 + POISSON)) * m["volume"] * scale[i], device="cuda", dtype=torch.float64)
            kappa = torch.full((t,), e / (3 * (1 - 2 * POISSON)) * m["volume"] * scale[i], device="cuda", dtype=torch.float64)
            x, v = _wide(g.positions), torch.zeros((m["n"], 3), device="cuda", dtype=torch.float64)
            poses = _wide(_capsules(g, seed + i, PRESS))
            for k in range(case["frames"]):
                x, v = _frame(m, x, v, mu, kappa, DT, case["substeps"], 1e6, 0.0, (poses[k], poses[k + 1]))
            out.append(x)
        return [torch.cat(out).cpu().numpy()]
    key = (case.get("spacing", SPACING), case["x"], case["y"], case["z"])
    grid = _grid(*key)
    if kind in ("step", "view"):
        m = _mesh(*key)
        e = YOUNG * METERS_PER_UNIT
        if case["x"] == 0:
            t = m["tets"].shape[0]
            mu = torch.full((t,), e / (2 * (1 + POISSON)) * m["volume"], device="cuda", dtype=torch.float64)
            kappa = torch.full((t,), e / (3 * (1 - 2 * POISSON)) * m["volume"], device="cuda", dtype=torch.float64)
        else:
            mu, kappa = (_wide(a) for a in _stiffness(grid, seed))
        x, v = (_wide(a) for a in _state_of(grid, seed))
        poses = None
        if case["tool"] == "capsule":
            poses = _wide(_capsules(grid, seed, PRESS))[:2]
        x, v = _frame(m, x, v, mu, kappa, 1 / 30 if case["x"] == 0 else DT, case["substeps"], case["ks"], case["damping"], poses)
        return [x.cpu().numpy(), None, None, None] if kind == "view" else [x.cpu().numpy(), v.cpu().numpy()]
    if case["frames"] * case["substeps"] * (3 if case["grad"] else 1) > 220:
        return None
    m = _mesh(*key)
    theta, path, target = _material(case, grid, seed)
    theta = _wide(theta).requires_grad_(case["grad"])
    path = _wide(path).requires_grad_(case["grad"])
    e = YOUNG * METERS_PER_UNIT * m["volume"] / (torch.exp(theta) * 1e6)
    mu, kappa = e / (2 * (1 + POISSON)), e / (3 * (1 - 2 * POISSON))
    x, v = _wide(grid.positions), torch.zeros((m["n"], 3), device="cuda", dtype=torch.float64)
    for k in range(case["frames"]):
        x, v = _frame(m, x, v, mu, kappa, DT, case["substeps"], 1e6, 0.0, (path[k], path[k + 1]))
    if not case["grad"]:
        return [x.cpu().numpy()]
    top = float(grid.positions[grid.active != 0, 1].max())
    at = torch.tensor(np.nonzero((grid.active != 0) & (np.abs(grid.positions[:, 1] - top) < 1e-6))[0], device="cuda")
    ((x[at] - _wide(target)[at]) ** 2).mean().backward()
    return [x.detach().cpu().numpy(), theta.grad.cpu().numpy(), path.grad.cpu().numpy()]
