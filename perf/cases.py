"""The workloads this repository is timed on, through its Python binding.

A *rollout* is what a training loop, a planner or a replay does with a batch
of worlds: rewind the batch to a stored state, step it, read the bodies back.
The state it rewinds to has run long enough that bodies have landed on each
other, so contacts dominate as they do in most of an episode.  A *query* asks
the narrowphase or the broadphase directly.

Sizes are those of the scenes in rbps_b200.scenes and of the tests, with odd
and uneven ones among them.
"""
import ctypes
import math

import numpy as np
import torch

import rbps_b200
from rbps_b200 import abi, scenes

FIELDS = ("position", "orientation", "linear_velocity", "angular_velocity")
PRECISION = {"fp64": abi.PRECISION_FP64, "fp32": abi.PRECISION_FP32, "fp32_pos64": abi.PRECISION_FP32_POS64}
ORDER = {"reference": abi.SOLVE_REFERENCE_ORDER, "colored": abi.SOLVE_COLORED}


def listed():
    return [
        # One World with the constructor's defaults (FP64, the reference's
        # order, 1/60 s, 20 substeps), an interactive scene of a few dozen
        # bodies: the smallest call, where launches and latency count.
        rollout("world_small", "pile", precision="fp64", order="reference", bodies=31, substeps=20, settle=60, steps=1),
        # The reference's plain scene: one world of 512 boxes and spheres,
        # FP64 in the reference's order, 10 substeps.
        rollout("world_plain", "pile", precision="fp64", order="reference", bodies=512, substeps=10, settle=60, steps=1),
        # A set of uneven worlds with jointed chains stepped in the
        # reference's order in FP64: parity runs and generated data.
        rollout("batch_reference", "uneven", precision="fp64", order="reference", worlds=96, bodies=128, substeps=4,
                settle=120, steps=2),
        # A few uneven worlds on the throughput path: evaluation of a policy,
        # too few worlds to fill the chip.
        rollout("batch_few", "uneven", precision="fp32", order="colored", worlds=61, bodies=512, substeps=4,
                settle=240, steps=2),
        # The headline workload: 4,096 uneven worlds with a revolute chain
        # each, forces in and poses out through page-locked host buffers
        # every step.
        rollout("batch_many", "uneven", precision="fp32", order="colored", worlds=4096, bodies=512, substeps=4,
                settle=240, steps=4, io=True),
        # Box towers 10 km from the origin, positions relative to a double
        # origin, masses alternating 1:1000, 20 substeps.
        rollout("towers_far", "towers", precision="fp32_pos64", order="colored", worlds=256, bodies=64, substeps=20,
                settle=20, steps=1),
        # One world of 65,536 spheres, boxes, capsules and convex hulls.
        rollout("world_large", "mixed", precision="fp32", order="colored", bodies=65536, substeps=10, settle=5,
                steps=1),
        # One world of hanging capsule chains on ball joints with a cone.
        rollout("world_chains", "hanging", precision="fp32", order="colored", bodies=33 * 625, substeps=8, settle=10,
                steps=1),
        # Many small worlds of hulls, ellipsoids, cylinders, cones, terrains
        # and meshes: GJK / EPA and the triangle routines.
        rollout("batch_shapes", "shapes", precision="fp32", order="colored", worlds=250, bodies=40, substeps=4,
                settle=40, steps=1),
        # Direct narrowphase tests of host-side shape pairs.
        {"name": "collide", "kind": "collide", "precision": "fp64", "pairs": 6000},
        # Broadphase frames of a host program: some objects move, update,
        # pairs back.
        {"name": "broadphase", "kind": "broadphase", "objects": 8191, "moved": 160},
        # The allocation-free pair query on boxes that are on the device.
        {"name": "sap_query", "kind": "sap_query", "objects": 1999},
    ]


def rollout(name, scene, precision, order, bodies, substeps, settle, steps, worlds=1, io=False):
    return {"name": name, "kind": "rollout", "scene": scene, "precision": precision, "order": order,
            "worlds": worlds, "bodies": bodies, "substeps": substeps, "settle": settle, "steps": steps, "io": io}


def spread(rng, lo, hi):
    """A whole number from [lo, hi], even over its logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    what = rng.choice(["pile", "uneven", "uneven_reference", "towers", "mixed", "hanging", "shapes", "collide",
                       "broadphase", "sap_query"])
    if what == "pile":
        c = rollout("", "pile", rng.choice(["fp64", "fp64", "fp32"]), "reference", spread(rng, 16, 512),
                    rng.choice([4, 8, 10, 20]), 60, 1)
    elif what == "uneven":
        c = rollout("", "uneven", "fp32", "colored", spread(rng, 32, 512), 4, 120, rng.randint(1, 4),
                    worlds=spread(rng, 16, 2048), io=rng.random() < 0.5)
    elif what == "uneven_reference":
        c = rollout("", "uneven", rng.choice(["fp64", "fp32"]), "reference", spread(rng, 32, 128), 4, 120, 1,
                    worlds=spread(rng, 8, 128))
    elif what == "towers":
        c = rollout("", "towers", rng.choice(["fp32", "fp32_pos64"]), "colored", rng.randint(8, 64), 20, 20, 1,
                    worlds=spread(rng, 16, 256))
    elif what == "mixed":
        c = rollout("", "mixed", "fp32", "colored", spread(rng, 4500, 65536), 10, 5, 1)
    elif what == "hanging":
        c = rollout("", "hanging", "fp32", "colored", 33 * spread(rng, 140, 625), 8, 10, 1)
    elif what == "shapes":
        c = rollout("", "shapes", rng.choice(["fp64", "fp32"]), "colored", rng.randint(16, 48), 4, 40, 1,
                    worlds=spread(rng, 10, 250))
    elif what == "collide":
        c = {"kind": "collide", "precision": rng.choice(["fp64", "fp32"]), "pairs": spread(rng, 200, 20000)}
    elif what == "broadphase":
        n = spread(rng, 500, 16384)
        c = {"kind": "broadphase", "objects": n, "moved": max(1, n // 50)}
    else:
        c = {"kind": "sap_query", "objects": spread(rng, 200, 8192)}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ scenes
def build_scene(case, seed):
    kind, n, worlds = case["scene"], case["bodies"], case["worlds"]
    if kind == "pile":
        return scenes.Scene("pile", 1.0 / 60.0, case["substeps"], 0, [scenes.small_world(seed, n)])
    if kind == "uneven":
        return uneven_worlds(seed, worlds, n)
    if kind == "towers":
        return scenes.config4(seed, n_worlds=worlds, height=n)
    if kind == "mixed":
        # the density of the 65,536-body scene at every size
        return scenes.config1(seed, n_bodies=n, n_hull_shapes=64, extent=200.0 * (n / 65536.0) ** (1.0 / 3.0))
    if kind == "hanging":
        return scenes.config2(seed, n_chains=n // 33)
    specs = []
    makers = (scenes.hull_world, scenes.round_world, scenes.terrain_world, scenes.hull_world, scenes.mesh_world)
    for w in range(worlds):
        specs.append(makers[w % len(makers)](seed=seed * 4099 + w, n=n))
    return scenes.Scene("shapes", 1.0 / 60.0, case["substeps"], 0, specs)


def uneven_counts(worlds, n):
    """Boxes and spheres of each world, log-uniform in [8, n]; the same for
    every seed, so that a case always has the same bodies."""
    rng = np.random.Generator(np.random.PCG64(worlds))
    return np.clip(np.exp(rng.uniform(math.log(8), math.log(n + 1), worlds)).astype(int), 8, n)


def uneven_worlds(seed, worlds, n):
    """scenes.config3: boxes and spheres, a 13-link revolute capsule chain
    and a ground plane in every world, 1/120 s, 4 substeps."""
    rng = np.random.Generator(np.random.PCG64(seed))
    specs = []
    for count in uneven_counts(worlds, n):
        bodies, forces, colliders = scenes.box_sphere_world(rng, int(count))
        joints = []
        scenes.capsule_chain(bodies, forces, colliders, joints,
                             (rng.uniform(-4.5, -3.5), rng.uniform(1.0, 21.0), rng.uniform(-5.0, 5.0)))
        specs.append(scenes.WorldSpec(np.array(bodies, abi.BODY_DT), np.array(forces, np.float64),
                                      np.array(colliders, abi.COLLIDER_DT), np.array(joints, abi.JOINT_DT)))
    return scenes.Scene("uneven", 1.0 / 120.0, 4, 0, specs)


def prepare(case, seed):
    if case["kind"] == "collide":
        return prepare_collide(case, seed)
    if case["kind"] == "broadphase":
        return prepare_broadphase(case, seed)
    if case["kind"] == "sap_query":
        return prepare_sap_query(case, seed)
    scene = build_scene(case, seed)
    b = rbps_b200.Batch.from_scene(scene, PRECISION[case["precision"]], ORDER[case["order"]],
                                   max_pairs_per_world=1 << 20 if case["scene"] == "hanging" else 0)
    b.step(case["settle"])
    slot = b.snapshot()
    b.synchronize()
    s = {"case": case, "batch": b, "slot": slot}
    if case["io"]:
        n = scene.n_bodies
        force = np.concatenate([w.forces for w in scene.worlds])
        s["force"] = torch.from_numpy(force).pin_memory()
        s["position"] = torch.zeros((n, 3), dtype=torch.float64).pin_memory()
        s["orientation"] = torch.zeros((n, 4), dtype=torch.float64).pin_memory()
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "collide":
        return run_collide(s)
    if kind == "broadphase":
        return run_broadphase(s)
    if kind == "sap_query":
        return run_sap_query(s)
    b = s["batch"]
    b.restore(s["slot"])
    if s["case"]["io"]:
        for _ in range(s["case"]["steps"]):
            b.step_io_async(s["force"].data_ptr(), s["position"].data_ptr(), s["orientation"].data_ptr())
        b.synchronize()
        return {"position": s["position"], "orientation": s["orientation"]}
    b.step(s["case"]["steps"])
    return b.state_all(FIELDS)


# ----------------------------------------------------------------- queries
ROUND = (abi.SHAPE_SPHERE, abi.SHAPE_BOX, abi.SHAPE_CAPSULE)  # met by a sphere in the first half


def prepare_collide(case, seed):
    """Half the pairs are a sphere against a sphere, a box or a capsule, the
    other half any two of box, capsule, ellipsoid, cylinder, cone and hull.
    Centres are about a shape apart, so roughly half of them touch."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n = case["pairs"]
    b = rbps_b200.Batch(1, 1.0 / 60.0, 1, PRECISION[case["precision"]])
    hulls = []
    for _ in range(6):
        d = rng.standard_normal((int(rng.integers(16, 33)), 3))
        pts = d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.2, 0.6, 3)
        hulls.append(b.add_hull(pts, rbps_b200.quickhull(pts)))
    b.add_world(0, scenes.small_world(seed, 4))
    b.commit()
    half = n // 2
    wide = np.array([abi.SHAPE_BOX, abi.SHAPE_CAPSULE, abi.SHAPE_ELLIPSOID, abi.SHAPE_CYLINDER, abi.SHAPE_CONE,
                     abi.SHAPE_CONVEX_HULL])

    def side(kinds):
        c = np.zeros(n, abi.COLLIDER_DT)
        c["shape"] = kinds
        c["params"][:, :3] = rng.uniform(0.2, 0.5, (n, 3))
        c["hull"] = np.where(kinds == abi.SHAPE_CONVEX_HULL, rng.choice(hulls, n), 0)
        c["local_rot"][:, 0] = 1.0
        tf = np.zeros((n, 7))
        tf[:, :3] = rng.uniform(-0.45, 0.45, (n, 3))
        tf[:, 3:] = scenes.random_quats(rng, n)
        return c, tf

    first = np.arange(n) < half
    a, ta = side(np.where(first, abi.SHAPE_SPHERE, rng.choice(wide, n)))
    c, tc = side(np.where(first, rng.choice(ROUND, n), rng.choice(wide, n)))
    return {"case": case, "batch": b, "a": a, "ta": ta, "b": c, "tb": tc, "half": half}


def run_collide(s):
    m = s["batch"].collide(s["a"], s["ta"], s["b"], s["tb"])
    h = s["half"]
    return {name: {f: m[f][part] for f in ("status", "n_points", "normal", "position", "depth")}
            for name, part in (("round", slice(0, h)), ("convex", slice(h, None)))}


def random_boxes(rng, n):
    """n boxes at the density of the 65,536-body scene."""
    edge = 200.0 * (n / 65536.0) ** (1.0 / 3.0)
    lo = rng.uniform(0.0, edge, (n, 3))
    return np.concatenate([lo, lo + rng.uniform(0.4, 1.2, (n, 3))], axis=1)


def prepare_broadphase(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    n = case["objects"]
    boxes = random_boxes(rng, n)
    bp = rbps_b200.BroadPhase()
    handles = [bp.insert(i, boxes[i]) for i in range(n)]
    bp.update()
    who = rng.permutation(n)[:case["moved"]]
    there = boxes + np.tile(rng.normal(0.0, 1.0, (n, 3)), 2)
    return {"case": case, "bp": bp, "frames": [[(handles[i], at[i]) for i in who] for at in (there, boxes)],
            "pairs": [np.zeros((4 * n + 64, 2), np.int32) for _ in range(2)]}


def run_broadphase(s):
    """Two frames: the moving objects go over and come back.  The pairs of
    each go to the program's own buffer, -1 behind the last."""
    bp = s["bp"]
    for frame, kept in zip(s["frames"], s["pairs"]):
        for handle, box in frame:
            bp.move(handle, box)
        bp.update()
        pairs = bp.pairs()
        kept[:len(pairs)] = pairs
        kept[len(pairs):] = -1
    return s["pairs"]


def prepare_sap_query(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    n = case["objects"]
    return {"case": case, "boxes": torch.from_numpy(random_boxes(rng, n)).cuda(),
            "ids": torch.arange(n, dtype=torch.int32, device="cuda"),
            "pairs": torch.zeros((4 * n + 64, 2), dtype=torch.int32, device="cuda"),
            "count": torch.zeros(1, dtype=torch.int32, device="cuda")}


def run_sap_query(s):
    rc = rbps_b200.lib().rbps_sap_pairs_static(
        s["boxes"].data_ptr(), s["ids"].data_ptr(), len(s["ids"]), s["pairs"].data_ptr(), len(s["pairs"]),
        s["count"].data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise RuntimeError("rbps_sap_pairs_static: %d" % rc)
    return {"pairs": s["pairs"], "count": s["count"]}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: every body's state, mass properties, force and shape read once
    and its state written once a pass, and what a query reads and returns.
    Flops: what a body costs a substep (integration, velocity update and
    about two contact points in both solves, a contact point about 900), a
    narrowphase test, a comparison per endpoint and sorting step."""
    if case["kind"] == "collide":
        return {"bytes": case["pairs"] * (2 * (136 + 56) + 160), "flops": case["pairs"] * 2000}
    if case["kind"] == "broadphase":
        n = case["objects"]
        return {"bytes": 2 * (n * (48 + 4) + 8 * n), "flops": 2 * 2 * n * 8}
    if case["kind"] == "sap_query":
        n = case["objects"]
        return {"bytes": n * (48 + 4) + 8 * n, "flops": 2 * n * 8}
    size = 8 if case["precision"] == "fp64" else 4
    bodies = case["bodies"] * case["worlds"]
    if case["scene"] == "uneven":  # and the chain and the ground
        bodies = int(uneven_counts(case["worlds"], case["bodies"]).sum()) + 14 * case["worlds"]
    b = bodies * (size * (16 + 12 + 3 + 3 + 13) + 96)
    if case["io"]:
        b += bodies * case["steps"] * 8 * (3 + 7)
    return {"bytes": b, "flops": bodies * case["substeps"] * case["steps"] * 2000}


# ------------------------------------------------------------------- exact
def rotate(q, v):
    w, u = q[:, :1], q[:, 1:]
    t = 2.0 * np.cross(u, v)
    return v + w * t + np.cross(u, t)


def exact_round(s):
    """The manifolds of the sphere pairs: one point, the deepest, on the
    second shape (a sphere pair's on the first); the normal from the first
    shape to the second."""
    h = s["half"]
    a, ta, b, tb = s["a"][:h], s["ta"][:h], s["b"][:h], s["tb"][:h]
    conj = tb[:, 3:] * np.array([1.0, -1.0, -1.0, -1.0])
    r, x = a["params"][:, 0], rotate(conj, ta[:, :3] - tb[:, :3])  # the sphere in the other's frame
    p = b["params"]
    ball, box = b["shape"] == abi.SHAPE_SPHERE, b["shape"] == abi.SHAPE_BOX
    near = np.where(box[:, None], np.clip(x, -p[:, :3], p[:, :3]), 0.0)  # nearest point of the box / core
    near[:, 1] = np.where(ball | box, near[:, 1], np.clip(x[:, 1], -p[:, 0], p[:, 0]))
    skin = np.where(box, 0.0, np.where(ball, p[:, 0], p[:, 1]))
    d = x - near
    dist = np.linalg.norm(d, axis=1)
    inside = box & (dist <= 1e-9)
    out = d / np.where(dist > 1e-9, dist, 1.0)[:, None]
    depth = r + skin - dist
    room = p[:, :3] - np.abs(x)
    k = np.argmin(room, axis=1)
    face = np.where(np.arange(3) == k[:, None], np.where(x > 0.0, 1.0, -1.0), 0.0)
    out = np.where(inside[:, None], face, out)
    near = np.where(inside[:, None] & (face != 0.0), face * p[:, :3], near)
    depth = np.where(inside, r + room.min(axis=1), depth)
    at = np.where(ball[:, None], x - out * r[:, None], near + out * skin[:, None])
    hit = depth > 0.0
    normal, pos, dep = np.zeros((h, 3)), np.zeros((h, 4, 3)), np.zeros((h, 4))
    normal[hit] = -rotate(tb[:, 3:], out)[hit]
    pos[hit, 0] = (tb[:, :3] + rotate(tb[:, 3:], at))[hit]
    dep[hit, 0] = depth[hit]
    return {"status": None, "n_points": None, "normal": normal, "position": pos, "depth": dep}


def exact(case, seed):
    """Only the direct narrowphase tests of round shapes have a value in
    closed form.  A step's result is that of an iteration in a stated order
    whose contact set hangs on every rounding; its value is the engine's."""
    if case["kind"] != "collide":
        return None
    none = {"status": None, "n_points": None, "normal": None, "position": None, "depth": None}
    return {"round": exact_round(prepare_collide(case, seed)), "convex": none}
