"""Performance cases of the framework: what its users run, over the sizes they run it at.

Kinds (each case names one):

* ``frame``      one resident scene advanced for a viewer or a controller: the packed body state
                 goes up from pinned host memory, the scene steps a few times, the state comes
                 back (``GpuScene.step_io``).  Small scenes are bound by latency and launches.
* ``pile``       the large pile of cubes, rods and voxelised spheres, the same call, grid or BVH
                 broad phase: throughput.
* ``batch``      many independent scenes of mixed sizes advanced together (``Batch.step``), every
                 scene's state read back: parameter sweeps, served requests.
* ``lbvh``       a tree over a point set through the stage entry points: scene box, Morton codes
                 (30 or 63 bits), radix sort, Karras hierarchy, leaves, refit.
* ``sis``        the sequential-impulse path, the reference's default update (``SISScene.step``).
* ``stages``     the reference's DEM step through the drop-in stage entry points, uniform grid
                 (updateUniformGridDEM with the wall collisions) or BVH (updateRigidBodies).
* ``depth``      an augmented-reality frame: depth image -> point cloud and normals -> attached to
                 a resident scene -> a few steps with the cloud as an obstacle -> state back.

A pass always starts from the case's own initial state, so every pass does the same work.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from diploma_thesis_b200 import api, scenes, sis
from diploma_thesis_b200._lib import call
from diploma_thesis_b200.api import ptr, stream_handle


def listed() -> list[dict]:
    return [
        # a toy scene in a viewer or a control loop, one step per frame: pure latency
        {"name": "frame_small", "kind": "frame", "layout": "packed", "side": 4, "edge": 3,
         "broadphase": "grid", "steps": 1},
        # the plain single-scene configuration (4,096 cubes of 27), ten steps per frame
        {"name": "frame_plain", "kind": "frame", "layout": "lattice", "side": 16, "edge": 3,
         "broadphase": "grid", "steps": 10},
        # the headline configuration, 2,097,152 particles
        {"name": "pile_grid", "kind": "pile", "bodies": 32768, "broadphase": "grid", "steps": 10},
        # the same pile through the BVH broad phase
        {"name": "pile_bvh", "kind": "pile", "bodies": 32768, "broadphase": "bvh", "steps": 5},
        # a sweep over scenes of 2k to 200k particles
        {"name": "batch_grid", "kind": "batch", "scenes": 40, "low": 2000, "high": 200000,
         "broadphase": "grid", "steps": 10},
        # a batch of BVH scenes (64-bit keys: more than four scenes)
        {"name": "batch_bvh", "kind": "batch", "scenes": 12, "low": 2000, "high": 100000,
         "broadphase": "bvh", "steps": 10},
        # the LBVH microbenchmark's largest size: clustered points with exact duplicates
        {"name": "lbvh_16m", "kind": "lbvh", "points": 1 << 24, "dist": "gmm", "bits": 30},
        # an ordinary, odd size with the fine codes
        {"name": "lbvh_63", "kind": "lbvh", "points": 1000003, "dist": "uniform", "bits": 63},
        # the sequential-impulse benchmark scene: 4,096 packed cubes of 27
        {"name": "sis_packed", "kind": "sis", "side": 16, "edge": 3, "steps": 1},
        # a program ported from the reference's wrappers, uniform grid, 13,824 packed cubes
        {"name": "stages_grid", "kind": "stages", "side": 24, "edge": 3, "broadphase": "grid",
         "steps": 1},
        # the same through the BVH, an odd size
        {"name": "stages_bvh", "kind": "stages", "side": 17, "edge": 3, "broadphase": "bvh",
         "steps": 1},
        # a depth-camera frame at the sensor's full resolution
        {"name": "depth_vga", "kind": "depth", "width": 640, "height": 480, "bodies": 400,
         "steps": 4},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(["frame", "frame", "pile", "pile", "batch", "batch", "lbvh", "lbvh", "sis",
                       "stages", "stages", "depth"])
    if kind == "frame":
        return {"kind": kind, "layout": rng.choice(["packed", "lattice"]),
                "side": rng.randint(2, 16), "edge": rng.choice([2, 3, 3, 4]),
                "broadphase": rng.choice(["grid", "bvh"]), "steps": rng.randint(1, 10)}
    if kind == "pile":
        bodies = _log_int(rng, 500, 32768)
        bvh = rng.random() < 0.5
        return {"kind": kind, "bodies": bodies, "broadphase": "bvh" if bvh else "grid",
                "steps": rng.randint(2, 5 if bvh else 10)}
    if kind == "batch":
        bvh = rng.random() < 0.5
        low = _log_int(rng, 1000, 4000)
        return {"kind": kind, "scenes": rng.randint(2, 12 if bvh else 40), "low": low,
                "high": low * rng.randint(2, 25 if bvh else 50),
                "broadphase": "bvh" if bvh else "grid", "steps": rng.randint(2, 10)}
    if kind == "lbvh":
        bits = rng.choice([30, 30, 63])
        return {"kind": kind, "points": _log_int(rng, 2000, 1 << 24 if bits == 30 else 1 << 22),
                "dist": rng.choice(["uniform", "gmm"]), "bits": bits}
    if kind == "sis":
        return {"kind": kind, "side": rng.randint(3, 15), "edge": rng.choice([2, 3]), "steps": 1}
    if kind == "stages":
        bvh = rng.random() < 0.5
        return {"kind": kind, "side": rng.randint(4, 17 if bvh else 24), "edge": 3,
                "broadphase": "bvh" if bvh else "grid", "steps": 1}
    return {"kind": kind, "width": rng.randint(160, 640), "height": rng.randint(120, 480),
            "bodies": _log_int(rng, 20, 400), "steps": rng.randint(1, 4)}


# ---- inputs -------------------------------------------------------------------------------------
STATE = ("body_pos", "body_quat", "body_vel", "body_angvel")


def _packed_state(sc: scenes.Scene) -> np.ndarray:
    return np.stack([getattr(sc, k) for k in STATE]).astype(np.float32)


def _pinned(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def _cubes(side: int, edge: int, layout: str, seed: int) -> scenes.Scene:
    """side^3 cubes of edge^3 particles: the plain configuration's jittered lattice over the unit
    box, or packed so that neighbours are in contact from the first step."""
    r = 1.0 / 256 if layout == "lattice" else 1.0 / (2.5 * side * edge)
    if layout == "packed":
        return scenes.small_scene(seed, nb_side=side, k=edge, r=r, packed=True)
    if edge == 3:
        return scenes.config0(seed, lattice=side)
    return scenes.small_scene(seed, nb_side=side, k=edge, r=min(r, 1.0 / (4 * side * edge)))


def _scene(case: dict, seed: int) -> scenes.Scene:
    if case["kind"] == "pile":
        return scenes.config2(seed, num_bodies=case["bodies"])
    return _cubes(case["side"], case["edge"], case["layout"], seed)


def _batch_scenes(case: dict, seed: int) -> list[scenes.Scene]:
    """Particle counts spread over the logarithm of the range, box sides over [0.5, 2]."""
    rng = np.random.default_rng(seed)
    counts = np.geomspace(case["low"], case["high"], case["scenes"])
    sides = 0.5 + 1.5 * ((np.arange(case["scenes"]) * 0.618) % 1.0)
    return [scenes.cube_scene(int(rng.integers(1 << 31)), int(c), float(s))
            for c, s in zip(counts, sides)]


# the depth camera's model (the loader's fixed intrinsics and gravity vector)
FOCAL, CENTRE = (517.3, 516.5), (318.6, 255.3)
GRAVITY = np.array([0.478957, -8.010560, 4.166928])
DEPTH_RADIUS = 1.0 / 128


def _depth_image(case: dict, seed: int) -> np.ndarray:
    """A wavy surface about a metre away (5,000 units per metre) with a hole without depth."""
    rng = np.random.default_rng(seed)
    h, w = case["height"], case["width"]
    y, x = np.mgrid[0:h, 0:w]
    a, b, c = rng.uniform(0.0, 2 * np.pi, 3)
    z = (1.0 + 0.10 * np.sin(x / 97.0 + a) + 0.08 * np.cos(y / 71.0 + b)
         + 0.02 * np.sin((x + y) / 23.0 + c) + rng.normal(0.0, 2e-4, (h, w)))
    hx, hy = int(rng.integers(0, w - w // 8)), int(rng.integers(0, h - h // 8))
    z[hy:hy + h // 8, hx:hx + w // 8] = 0.0
    return np.clip(z * 5000.0, 0, 32767).astype(np.int16)


def _depth_cloud(depth: np.ndarray):
    """Cloud and normals of a depth image in 64 bits, with the loader's rules: a pixel without
    depth lies at z = -1000, the last width + height - 2 pixels and the border normals stay 0."""
    h, w = depth.shape
    y, x = np.mgrid[0:h, 0:w].astype(np.float64)
    z = depth / 5000.0
    z = np.where(z < 0.01, -1000.0, z)
    px, py = z * (x - CENTRE[0]) / FOCAL[0], z * (y - CENTRE[1]) / FOCAL[1]
    gx, gy, gz = GRAVITY / np.linalg.norm(GRAVITY)
    pos = np.stack([px - gx * py, gy * py - gz * z, gz * py + gy * z], -1)
    pos.reshape(-1, 3)[(w - 1) * (h - 1) + 1:] = 0.0
    nrm = np.zeros_like(pos)
    c = np.cross(pos[2:, 1:-1] - pos[:-2, 1:-1], pos[1:-1, 2:] - pos[1:-1, :-2])
    length = np.linalg.norm(c, axis=-1, keepdims=True)
    nrm[1:-1, 1:-1] = np.where(length > 0, c / np.where(length > 0, length, 1.0), 0.0)
    return pos.reshape(-1, 3), nrm.reshape(-1, 3)


def _depth_scene(case: dict, seed: int, depth: np.ndarray) -> scenes.Scene:
    """Small cubes dropped onto the camera's surface."""
    pos, nrm = _depth_cloud(depth)
    rng = np.random.default_rng(seed + 1)
    good = (np.abs(pos).max(1) < 10.0) & (np.abs(np.linalg.norm(nrm, axis=1) - 1) < 1e-3)
    pick = rng.choice(np.flatnonzero(good), case["bodies"], replace=False)
    r = DEPTH_RADIUS
    centres = pos[pick] + 2.5 * r * nrm[pick]
    sc = scenes._assemble([scenes.cube_body(2, 2 * r)] * len(pick), centres,
                          scenes.random_quaternions(rng, len(pick)),
                          rng.normal(0.0, 0.2, (len(pick), 3)), r, pos[good].min(0) - 0.1,
                          pos[good].max(0) + 0.1, name="cubes on a depth-camera surface")
    sc.spring = 500.0  # many cloud points touch a particle at once
    return sc


class State:
    """What a program keeps between calls; resident scenes are closed with it."""

    def __init__(self, case: dict):
        self.case = case
        self.ctx = api.Context(0)
        self.resident: list = []

    def __del__(self):
        for r in self.resident:
            r.close()
        self.ctx.close()


def prepare(case: dict, seed: int) -> State:
    s = State(case)
    globals()["_prepare_" + case["kind"]](s, case, seed)
    return s


def _prepare_frame(s: State, case: dict, seed: int) -> None:
    sc = _scene(case, seed)
    s.scene = api.GpuScene(s.ctx, sc, broadphase=case["broadphase"])
    s.resident.append(s.scene)
    s.pinned = _pinned(_packed_state(sc)), _pinned(np.zeros((4, sc.num_bodies, 4), np.float32))
    s.up, s.down = (t.numpy() for t in s.pinned)


_prepare_pile = _prepare_frame


def _prepare_batch(s: State, case: dict, seed: int) -> None:
    many = _batch_scenes(case, seed)
    s.members = [api.GpuScene(s.ctx, sc, broadphase=case["broadphase"]) for sc in many]
    s.batch = api.Batch(s.ctx, s.members)
    s.resident += [s.batch, *s.members]
    s.pinned = [(_pinned(_packed_state(sc)),
                 _pinned(np.zeros((4, sc.num_bodies, 4), np.float32))) for sc in many]
    s.up = [a.numpy() for a, _ in s.pinned]
    s.down = [b.numpy() for _, b in s.pinned]


def _prepare_lbvh(s: State, case: dict, seed: int) -> None:
    n = case["points"]
    s.pos = torch.from_numpy(scenes.lbvh_points(n, case["dist"], seed)).cuda()
    s.tree = _tree_buffers(n, case["bits"])


def _tree_buffers(n: int, bits: int) -> dict[str, torch.Tensor]:
    def z(count, dtype=torch.int32):
        return torch.zeros(count, dtype=dtype, device="cuda")
    key = torch.int32 if bits == 30 else torch.int64
    m = 2 * n - 1
    return {"lo": z(4, torch.float32), "hi": z(4, torch.float32), "codes": z(n, key),
            "idx": z(n), "sorted": z(n, key), "order": z(n), "leaf": z(m, torch.uint8),
            "left": z(m), "right": z(m), "parent": z(m), "min_r": z(m), "max_r": z(m),
            "cms": z((n, 4), torch.float32), "bounds": z((m, 8), torch.float32),
            "radii": z(n, torch.float32)}


def _prepare_sis(s: State, case: dict, seed: int) -> None:
    sc = _cubes(case["side"], case["edge"], "packed", seed)
    s.sis = sis.SISScene(s.ctx, sc, sc.dt)
    s.first = {k: getattr(s.sis, k).clone() for k in ("cms", "vel", "ang", "quat", "rel")}


def _stage_arrays(case: dict, seed: int):
    """A packed scene in the reference's layouts and units (impulse per step, world-frame particle
    offsets), in a box whose walls cut into the outermost bodies."""
    sc = _cubes(case["side"], case["edge"], "packed", seed)
    rel = np.zeros((sc.num_particles, 4), np.float32)
    world = sc.world_positions()
    rel[:, :3] = world[:, :3] - sc.body_pos[sc.body_index(), :3]
    rng = np.random.default_rng(seed + 1)
    ang = np.zeros((sc.num_bodies, 4), np.float32)
    ang[:, :3] = rng.normal(0.0, 1.0, (sc.num_bodies, 3))
    r = np.float32(sc.radius)
    return sc, rel, ang, world[:, :3].min(0) + r / 4, world[:, :3].max(0) - r / 4


F32 = C.POINTER(C.c_float)
STAGE_DT = 1e-3
STAGE_LAW = {"spring": 0.5, "damping": 0.02, "shear": 0.1, "attraction": 0.0}
STAGE_GRAVITY = (0.0, -9.81e-3, 0.0)  # added to the velocity once per step


def _prepare_stages(s: State, case: dict, seed: int) -> None:
    sc, rel, ang, lo, hi = _stage_arrays(case, seed)
    n, nb = sc.num_particles, sc.num_bodies

    def dev(a, dtype=torch.float32):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dtype).cuda()

    def z(shape, dtype=torch.float32):
        return torch.zeros(shape, dtype=dtype, device="cuda")

    s.n, s.nb, s.radius = n, nb, float(sc.radius)
    cells = 1 << max(2, math.ceil(math.log2(1.0 / (2 * sc.radius))))
    s.cells = cells ** 3
    s.params = api.sim_params(sc.radius, (0.0, 0.0, 0.0), 2 * float(sc.radius), (cells,) * 3,
                              gravity=STAGE_GRAVITY, **STAGE_LAW)
    s.lo, s.hi = (np.ascontiguousarray(a, np.float32) for a in (lo, hi))
    s.first = {"cms": dev(sc.body_pos), "vel": dev(sc.body_vel), "ang": dev(ang),
               "rel": dev(rel), "cum": dev(sc.body_quat)}
    s.b = {k: v.clone() for k, v in s.first.items()}
    s.b |= {"quat": z((nb, 4)), "ib": dev(sc.body_inv_inertia), "cur": z((nb, 9)),
            "model": z((nb, 16)), "mass": dev(sc.body_mass),
            "offsets": dev(sc.body_offsets, torch.int32), "rb": dev(sc.body_index(), torch.int32),
            "pos": z((n, 4)), "pvel": z((n, 4)), "force": z((n, 4)), "torque": z((n, 4))}
    if case["broadphase"] == "grid":
        i32 = torch.int32
        s.b |= {"hash": z(n, i32), "idx": z(n, i32), "shash": z(n, i32), "sidx": z(n, i32),
                "start": z(s.cells, i32), "end": z(s.cells, i32), "spos": z((n, 4)),
                "svel": z((n, 4))}
    else:
        s.tree = _tree_buffers(n, 30)


def _prepare_depth(s: State, case: dict, seed: int) -> None:
    depth = _depth_image(case, seed)
    sc = _depth_scene(case, seed, depth)
    s.depth = torch.from_numpy(depth).cuda()
    s.camera = np.eye(4, dtype=np.float32).reshape(16)
    m = case["width"] * case["height"]
    s.pos, s.norm = (torch.zeros((m, 4), device="cuda") for _ in range(2))
    s.radii = torch.zeros(m, device="cuda")
    s.scene = api.GpuScene(s.ctx, sc)
    s.resident.append(s.scene)
    s.pinned = _pinned(_packed_state(sc)), _pinned(np.zeros((4, sc.num_bodies, 4), np.float32))
    s.up, s.down = (t.numpy() for t in s.pinned)


# ---- one pass -----------------------------------------------------------------------------------
def run(state: State):
    return globals()["_run_" + state.case["kind"]](state, state.case)


def _run_frame(s: State, case: dict):
    s.scene.step_io(s.up, case["steps"], s.down)
    return s.down


_run_pile = _run_frame


def _run_batch(s: State, case: dict):
    for g, up in zip(s.members, s.up):
        g.upload_state(up)
    s.batch.step(case["steps"])
    for g, down in zip(s.members, s.down):
        g.download_state(down, wait=False)
    torch.cuda.current_stream().synchronize()  # the states are on the host from here on
    return s.down


def _build_tree(s: State, pos: torch.Tensor, n: int, bits: int, radius: float, st) -> None:
    t, h = s.tree, s.ctx.handle
    call("ar_scene_aabb", h, ptr(pos), n, ptr(t["lo"]), ptr(t["hi"]), st)
    name, width = ("ar_morton30", "32") if bits == 30 else ("ar_morton63", "64")
    call(name, h, ptr(pos), n, ptr(t["lo"]), ptr(t["hi"]), ptr(t["codes"]), ptr(t["idx"]), st)
    call("ar_radix_sort_pairs_u" + width, h, ptr(t["codes"]), ptr(t["idx"]), ptr(t["sorted"]),
         ptr(t["order"]), n, 0, bits, st)
    call("ar_lbvh_build" if bits == 30 else "ar_lbvh_build64", h, ptr(t["sorted"]), n,
         ptr(t["leaf"]), ptr(t["left"]), ptr(t["right"]), ptr(t["parent"]), ptr(t["min_r"]),
         ptr(t["max_r"]), st)
    call("ar_lbvh_leaves", h, n, ptr(t["order"]), ptr(pos), C.c_float(radius), ptr(t["leaf"]),
         ptr(t["min_r"]), ptr(t["max_r"]), ptr(t["cms"]), ptr(t["bounds"]), ptr(t["radii"]), st)
    call("ar_lbvh_refit", h, n, ptr(t["left"]), ptr(t["right"]), ptr(t["parent"]),
         ptr(t["bounds"]), st)


LBVH_RADIUS = 1e-3


def _run_lbvh(s: State, case: dict):
    _build_tree(s, s.pos, case["points"], case["bits"], LBVH_RADIUS, stream_handle())
    return {k: v for k, v in s.tree.items() if k not in ("idx", "cms", "radii")}


def _run_sis(s: State, case: dict):
    for k, v in s.first.items():
        getattr(s.sis, k).copy_(v)
    s.sis.step(case["steps"])
    return {k: getattr(s.sis, k) for k in ("cms", "vel", "ang", "cur", "rel", "pos", "pvel",
                                           "count")}


def _run_stages(s: State, case: dict):
    b, h, n, nb, st = s.b, s.ctx.handle, s.n, s.nb, stream_handle()
    prm = C.byref(s.params)
    for k, v in s.first.items():
        b[k].copy_(v)
    for _ in range(case["steps"]):
        call("ar_integrate_reference", h, prm, C.c_float(STAGE_DT), nb, ptr(b["cms"]),
             ptr(b["vel"]), ptr(b["ang"]), ptr(b["quat"]), ptr(b["ib"]), ptr(b["cur"]),
             ptr(b["model"]), ptr(b["cum"]), ptr(b["mass"]), st)
        call("ar_global_attributes", h, n, nb, ptr(b["cms"]), ptr(b["vel"]), ptr(b["ang"]),
             ptr(b["quat"]), ptr(b["rb"]), ptr(b["rel"]), ptr(b["pos"]), ptr(b["pvel"]), st)
        call("ar_reset_quaternions", h, ptr(b["quat"]), nb, st)
        if case["broadphase"] == "grid":
            call("ar_calc_hash", h, prm, ptr(b["pos"]), n, ptr(b["hash"]), ptr(b["idx"]), st)
            call("ar_radix_sort_pairs_u32", h, ptr(b["hash"]), ptr(b["idx"]), ptr(b["shash"]),
                 ptr(b["sidx"]), n, 0, 32, st)
            call("ar_reorder_cells", h, ptr(b["shash"]), ptr(b["sidx"]), ptr(b["pos"]),
                 ptr(b["pvel"]), n, s.cells, ptr(b["start"]), ptr(b["end"]), ptr(b["spos"]),
                 ptr(b["svel"]), st)
            call("ar_fill_f32", h, ptr(b["force"]), 4 * n, C.c_float(0.0), st)
            call("ar_fill_f32", h, ptr(b["torque"]), 4 * n, C.c_float(0.0), st)
            call("ar_collide_grid_dem", h, prm, ptr(b["rb"]), ptr(b["spos"]), ptr(b["svel"]),
                 ptr(b["rel"]), ptr(b["sidx"]), ptr(b["start"]), ptr(b["end"]), n,
                 ptr(b["force"]), ptr(b["torque"]), st)
        else:
            t = s.tree
            _build_tree(s, b["pos"], n, 30, s.radius, st)
            call("ar_collide_bvh_dem", h, prm, ptr(b["rb"]), ptr(b["rel"]), ptr(b["pvel"]),
                 ptr(t["leaf"]), ptr(t["left"]), ptr(t["right"]), ptr(t["parent"]),
                 ptr(t["cms"]), ptr(t["bounds"]), ptr(t["order"]), ptr(t["radii"]), n,
                 ptr(b["force"]), ptr(b["torque"]), None, st)
        call("ar_reduce_impulses", h, ptr(b["force"]), ptr(b["torque"]), ptr(b["offsets"]), nb,
             ptr(b["vel"]), ptr(b["ang"]), ptr(b["mass"]), ptr(b["ib"]), st)
        call("ar_walls_reference", h, C.c_float(s.radius), ptr(b["pos"]), ptr(b["cms"]),
             s.lo.ctypes.data_as(F32), s.hi.ctypes.data_as(F32), ptr(b["vel"]),
             ptr(b["ang"]), ptr(b["ib"]), ptr(b["mass"]), ptr(b["rb"]), ptr(b["offsets"]), nb, n,
             st)
    return {k: b[k] for k in ("cms", "vel", "ang", "rel", "cur", "cum", "model", "pos", "pvel",
                              "force", "torque")}


def _run_depth(s: State, case: dict):
    h, st, w, ht = s.ctx.handle, stream_handle(), case["width"], case["height"]
    call("ar_range_image_cloud", h, ptr(s.depth), w, ht, s.camera.ctypes.data_as(C.c_void_p),
         C.c_float(DEPTH_RADIUS), ptr(s.pos), ptr(s.radii), None, st)
    call("ar_range_image_normals", h, ptr(s.pos), w, ht, ptr(s.norm), st)
    torch.nan_to_num_(s.norm, nan=0.0, posinf=0.0, neginf=0.0)  # neighbours that coincide
    s.scene.set_static_cloud(s.pos, s.norm)
    s.scene.step_io(s.up, case["steps"], s.down)
    return {"state": s.down, "pos": s.pos, "norm": s.norm}


# ---- the work a pass cannot do without ------------------------------------------------------------
def _step_work(n: int, nb: int) -> tuple[int, int]:
    """Bytes and operations of one step: particle offsets in, the body state in and out, mass and
    inverse inertia in; per particle its pose, 27 neighbour cells' tests and its share of the body
    sums, per body the integration."""
    return 16 * n + nb * (2 * 64 + 40), 150 * n + 200 * nb


def _tree_work(n: int, bits: int) -> tuple[int, int]:
    """Points in; box, sorted codes and order, the hierarchy's five links, flag and box per node,
    and the leaves' centres and radii out; per point its code, per node its split and its box."""
    m = 2 * n - 1
    return 16 * n + n * (2 * (4 if bits == 30 else 8) + 8) + m * 53 + n * 20, 150 * n


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "lbvh":
        b, f = _tree_work(case["points"], case["bits"])
    elif kind == "depth":
        m, nb = case["width"] * case["height"], case["bodies"]
        b, f = _step_work(8 * nb, nb)
        b, f = b * case["steps"] + m * (2 + 36), f * case["steps"] + 100 * m
    elif kind == "batch":
        # log-uniform particle counts, 27 to a body
        mean = (case["high"] - case["low"]) / math.log(case["high"] / case["low"])
        n = int(case["scenes"] * mean)
        b, f = _step_work(n, n // 27)
        b, f = b * case["steps"], f * case["steps"]
    else:
        if kind == "pile":
            nb, n = case["bodies"], 64 * case["bodies"]
        else:
            nb = case["side"] ** 3
            n = nb * case["edge"] ** 3
        b, f = _step_work(n, nb)
        if kind == "sis":  # about a contact per particle surface site, 18 sweeps of ~150 operations
            b, f = b + 48 * n, f + 18 * 150 * n
        elif kind == "stages":  # positions, velocities, forces and torques out as well
            b, f = b + 80 * n, f
            if case["broadphase"] == "bvh":
                tb, tf = _tree_work(n, 30)
                b, f = b + tb, f + tf
        b, f = b * case["steps"], f * case["steps"]
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits ------------------------------------------------------------------
def exact(case: dict, seed: int):
    """What run() returns, in 64-bit arithmetic by plain torch and numpy; None where that would
    take too long (the impulse solver's sequential sweeps)."""
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


def _device() -> str:
    return "cuda" if torch.cuda.is_available() else "cpu"


def _rotation(q: torch.Tensor) -> torch.Tensor:
    """Rotation matrices [B, 3, 3] of unit quaternions (x, y, z, w)."""
    x, y, z, w = q.unbind(-1)
    return torch.stack([
        1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)],
        -1).reshape(-1, 3, 3)


def _quat_mul(p: torch.Tensor, q: torch.Tensor) -> torch.Tensor:
    pv, pw, qv, qw = p[..., :3], p[..., 3:], q[..., :3], q[..., 3:]
    return torch.cat([pw * qv + qw * pv + torch.linalg.cross(pv, qv),
                      pw * qw - (pv * qv).sum(-1, keepdim=True)], -1)


def _near(a: torch.Tensor, b: torch.Tensor, reach: float):
    """For each of the 27 cell offsets, the (i, j) index pairs of points a_i, b_j in neighbouring
    cells of edge `reach` that are less than `reach` apart."""
    cell = reach * (1 + 1e-9)
    lo = torch.minimum(a.min(0).values, b.min(0).values) - cell
    top = torch.floor((torch.maximum(a.max(0).values, b.max(0).values) - lo) / cell).long() + 3

    def key(c):
        return (c[:, 2] * top[1] + c[:, 1]) * top[0] + c[:, 0]
    ca = torch.floor((a - lo) / cell).long()
    kb, order = torch.sort(key(torch.floor((b - lo) / cell).long()))
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = key(ca + torch.tensor([dx, dy, dz], device=a.device))
                first = torch.searchsorted(kb, k)
                count = torch.searchsorted(kb, k, right=True) - first
                i = torch.repeat_interleave(torch.arange(len(a), device=a.device), count)
                within = torch.arange(len(i), device=a.device) - (torch.cumsum(count, 0) - count)[i]
                j = order[first[i] + within]
                hit = ((b[j] - a[i]).square().sum(1) < reach * reach).nonzero()[:, 0]
                yield i[hit], j[hit]


def _law(rp, rv, normal, depth, k, damping, shear, attraction):
    rt = rv - (rv * normal).sum(1, keepdim=True) * normal
    return -k * depth * normal + damping * rv + shear * rt + attraction * rp


def _pair_forces(pos, vel, body, r, k, damping, shear, attraction):
    force = torch.zeros_like(pos)
    for i, j in _near(pos, pos, 2 * r):
        other = body[i] != body[j]
        i, j = i[other], j[other]
        rp = pos[j] - pos[i]
        d = rp.norm(dim=1, keepdim=True)
        force.index_add_(0, i, _law(rp, vel[j] - vel[i], rp / d, 2 * r - d, k, damping, shear,
                                    attraction))
    return force


def _cloud_forces(pos, vel, cloud, normals, r, k, damping, shear, attraction):
    force = torch.zeros_like(pos)
    for i, j in _near(pos, cloud, 2 * r):
        rp = cloud[j] - pos[i]
        d = rp.norm(dim=1, keepdim=True)
        force.index_add_(0, i, _law(rp, -vel[i], -normals[j], 2 * r - d, k, damping, shear,
                                    attraction))
    return force


def _exact_state(sc: scenes.Scene, steps: int, cloud=None) -> np.ndarray:
    """[4, B, 4] state of a scene after `steps` steps of the physical form."""
    dev = _device()

    def t(a):
        return torch.from_numpy(np.asarray(a, np.float64)).to(dev)
    pos, vel, ang = (t(getattr(sc, k)[:, :3]) for k in ("body_pos", "body_vel", "body_angvel"))
    quat, rel = t(sc.body_quat), t(sc.particle_rel[:, :3])
    body = torch.from_numpy(sc.body_index()).long().to(dev)
    mass = t(sc.body_mass)[:, None]
    inv = t(sc.body_inv_inertia).reshape(-1, 3, 3).transpose(1, 2)
    lo, hi, g = t(sc.box_min), t(sc.box_max), t(np.float32(sc.gravity))
    r, dt = float(np.float32(sc.radius)), float(np.float32(sc.dt))
    law = tuple(float(np.float32(v)) for v in (sc.spring, sc.damping, sc.shear, sc.attraction))
    for _ in range(steps):
        rot = _rotation(quat)
        arm = (rot[body] @ rel[:, :, None])[:, :, 0]
        p, v = pos[body] + arm, vel[body] + torch.linalg.cross(ang[body], arm)
        f = _pair_forces(p, v, body, r, *law)
        for a in range(3):
            for d, sign in ((p[:, a] - lo[a], 1.0), (hi[a] - p[:, a], -1.0)):
                hit = d < r
                rt = -v[hit]
                rt[:, a] = 0.0
                fw = law[1] * -v[hit] + law[2] * rt
                fw[:, a] += sign * law[0] * (r - d[hit])
                f[hit] += fw
        if cloud is not None:
            f += _cloud_forces(p, v, *cloud, r, *law)
        force = torch.zeros_like(pos).index_add_(0, body, f)
        torque = torch.zeros_like(pos).index_add_(0, body, torch.linalg.cross(arm, f))
        vel = vel + dt * (g + force / mass)
        world = rot @ inv @ rot.transpose(1, 2)
        ang = ang + dt * (world @ torque[:, :, None])[:, :, 0]
        pos = pos + dt * vel
        spin = torch.cat([ang, torch.zeros_like(mass)], 1)
        quat = quat + 0.5 * dt * _quat_mul(spin, quat)
        quat = quat / quat.norm(dim=1, keepdim=True)
    zero = torch.zeros_like(mass)
    out = [torch.cat([pos, zero], 1), quat, torch.cat([vel, zero], 1), torch.cat([ang, zero], 1)]
    return torch.stack(out).cpu().numpy()


def _exact_frame(case: dict, seed: int):
    return _exact_state(_scene(case, seed), case["steps"])


_exact_pile = _exact_frame


def _exact_batch(case: dict, seed: int):
    return [_exact_state(sc, case["steps"]) for sc in _batch_scenes(case, seed)]


def _exact_depth(case: dict, seed: int):
    depth = _depth_image(case, seed)
    pos, nrm = _depth_cloud(depth)
    cloud = tuple(torch.from_numpy(a).to(_device()) for a in (pos, nrm))
    four = [np.concatenate([a, np.zeros((len(a), 1))], 1) for a in (pos, nrm)]
    return {"state": _exact_state(_depth_scene(case, seed, depth), case["steps"], cloud),
            "pos": four[0], "norm": four[1]}


def _exact_lbvh(case: dict, seed: int):
    """The codes, the order and the hierarchy are whole numbers; the scene box is computed."""
    p = scenes.lbvh_points(case["points"], case["dist"], seed).astype(np.float64)
    out = dict.fromkeys(("codes", "sorted", "order", "leaf", "left", "right", "parent", "min_r",
                         "max_r", "bounds"))
    return out | {"lo": p.min(0), "hi": p.max(0)}


def _exact_stages(case: dict, seed: int):
    dev = _device()
    sc, rel, ang, lo, hi = _stage_arrays(case, seed)

    def t(a):
        return torch.from_numpy(np.asarray(a, np.float64)).to(dev)
    nb = sc.num_bodies
    cms, vel = t(sc.body_pos[:, :3]), t(sc.body_vel[:, :3])
    cum, mass = t(sc.body_quat), t(sc.body_mass)[:, None]
    ang, rel, lo, hi = t(ang[:, :3]), t(rel[:, :3]), t(np.float32(lo)), t(np.float32(hi))
    inv = t(sc.body_inv_inertia).reshape(-1, 3, 3).transpose(1, 2)
    body = torch.from_numpy(sc.body_index()).long().to(dev)
    r, dt = float(np.float32(sc.radius)), float(np.float32(STAGE_DT))
    law = tuple(float(np.float32(STAGE_LAW[k])) for k in ("spring", "damping", "shear",
                                                           "attraction"))
    one = torch.tensor([0.0, 0.0, 0.0, 1.0], dtype=torch.float64, device=dev)
    rows = torch.arange(nb, device=dev)
    for _ in range(case["steps"]):
        # integrate: position, rotation of the step, world inertia, orientation, gravity
        cms = cms + vel * dt
        speed = ang.norm(dim=1, keepdim=True)
        half = speed * dt / 2
        turn = torch.cat([torch.sin(half) * ang / speed.clamp_min(1e-300), torch.cos(half)], 1)
        turn = torch.where(2 * half > 1e-5, turn, one)
        rot = _rotation(turn)
        cur = rot @ inv @ rot.transpose(1, 2)
        cum = _quat_mul(turn, cum)
        cum = cum / cum.norm(dim=1, keepdim=True)
        vel = vel + t(np.float32(STAGE_GRAVITY))
        # particles
        rel = (rot[body] @ rel[:, :, None])[:, :, 0]
        pos, pvel = cms[body] + rel, vel[body] + torch.linalg.cross(ang[body], rel)
        force = _pair_forces(pos, pvel, body, r, *law)
        torque = torch.linalg.cross(rel, force)
        vel = vel + torch.zeros_like(vel).index_add_(0, body, force) / mass
        tb = torch.zeros_like(vel).index_add_(0, body, torque)
        ang = ang + (inv @ tb[:, :, None])[:, :, 0]
        # walls: a body's deepest particle past a wall it moves towards takes an elastic impulse
        depth = torch.cat([pos - hi + r, lo + r - pos], 1)  # +x, +y, +z, -x, -y, -z
        toward = torch.cat([vel, -vel], 1)[body] > 0
        depth, wall = torch.where(toward, depth, 0.0).max(1)
        deep = torch.zeros(nb, dtype=torch.float64, device=dev)
        deep.scatter_reduce_(0, body, depth, "amax")
        hit = (depth > 0) & (depth == deep[body])
        last = torch.full((nb,), -1, dtype=torch.long, device=dev)
        last.scatter_reduce_(0, body[hit], hit.nonzero()[:, 0], "amax")
        b = rows[last >= 0]
        w, p = wall[last[b]], pos[last[b]]
        n = torch.zeros((len(b), 3), dtype=torch.float64, device=dev)
        n[torch.arange(len(b), device=dev), w % 3] = torch.where(w < 3, 1.0, -1.0).double()
        plane = torch.where((w < 3)[:, None], hi, lo)
        moved = cms[b] + n.abs() * plane * n.abs() - r * n - n.abs() * p
        # the contact lies one radius from the particle along the wall's normal
        arm = moved - (moved + (p - cms[b]) + n * r)
        i_b, m_b = inv[b], mass[b, 0]
        va = vel[b] + torch.linalg.cross(ang[b], arm)
        lever = torch.linalg.cross((i_b @ torch.linalg.cross(arm, -n)[:, :, None])[:, :, 0], arm)
        j = (-2 * (va * -n).sum(1) / (1 / m_b + (lever * -n).sum(1)))[:, None]
        vel[b] += -n * j / mass[b]
        ang[b] += (i_b @ torch.linalg.cross(arm, -n * j)[:, :, None])[:, :, 0]

    def four(a):
        return torch.cat([a, torch.zeros_like(a[:, :1])], 1).cpu().numpy()
    model = torch.zeros((nb, 4, 4), dtype=torch.float64, device=dev)
    model[:, :3, :3] = _rotation(cum).transpose(1, 2)  # column-major
    model[:, 3, :3] = cms
    model[:, 3, 3] = 1.0
    return {"cms": four(cms), "vel": four(vel), "ang": four(ang), "rel": four(rel),
            "cur": cur.transpose(1, 2).reshape(nb, 9).cpu().numpy(), "cum": cum.cpu().numpy(),
            "model": model.reshape(nb, 16).cpu().numpy(), "pos": four(pos), "pvel": four(pvel),
            "force": four(force), "torque": four(torque)}
