"""The work that the performance of this framework is measured on: what programs built on it step,
through ``Sim``, ``Batch`` and ``Server``, from one small scene to thousands.

A pass advances a running simulation the way its program does (a viewer's frame, a policy's control
step, a wave of served requests) and returns what that program reads back. A state starts from a
settled scene; the seed draws the bodies' and joints' velocities, the joint targets and the
requests. The scenes themselves follow from the case alone, so they are built and settled once per
process and shared by its states.
"""
import copy
import math

import numpy as np

from steel_webgpu_b200 import SceneBuilder, pack, synth
from steel_webgpu_b200.sim import Batch, Server, Sim, auto_caps

TARGET_SETS = 8  # a control loop's pre-drawn joint targets, taken in turn


def listed():
    return [
        # A viewer or a test bench with a handful of boxes: one frame, the poses drawn.
        dict(name="app_boxes_12", kind="app", bodies=12, shapes="boxes", frames=1),
        # The smallest configured workload: 64 boxes on a plane, poses read every 4 frames.
        dict(name="app_boxes_64", kind="app", bodies=64, shapes="boxes", frames=4),
        # Every primitive and hulls, with the free bodies' torsional and rolling friction on.
        dict(name="app_mixed_77", kind="app", bodies=77, shapes="mixed", frames=1),
        # A bin of parts (hulls, boxes, capsules): one scene of ordinary size, full state read; the
        # builder's default contact gap, wide for parts of this size, so many rows and many colors.
        dict(name="pile_700", kind="pile", bodies=700, bin=3.0, gap=0.1, frames=1),
        # The plain method at scale: 8192 convex bodies settled in a bin, a gap that suits their size.
        dict(name="pile_8192", kind="pile", bodies=8192, bin=10.0, gap=0.02, frames=1),
        # One shared world of articulations: quadrupeds and 40-link chains, a control step of all.
        dict(name="herd_128_8", kind="herd", quads=128, chains=8, links=40, frames=1),
        # Reaching arms, a batch of independent scenes without contacts, two frames per action.
        dict(name="arms_1500", kind="arms", scenes=1500, links=7, frames=2),
        # Legged policy training: one quadruped per scene, one frame per action.
        dict(name="quads_1024", kind="quads", scenes=1024, frames=1, cone=""),
        # The same with articulated torsional and rolling friction (elliptic cone), a smaller batch.
        dict(name="quads_cone_96", kind="quads", scenes=96, frames=1, cone="elliptic"),
        # Continuous batching: resident instances of mixed sizes, a wave of requests served to the end.
        dict(name="serve_320", kind="serve", scenes=320, requests=64),
        # The uneven batch of box piles and chains, small and on the default tiles.
        dict(name="uneven_256", kind="uneven", scenes=256, fp64=False, tuned=False),
        # The headline workload: 2048 uneven scenes, FP64 articulated inertia, autotuned tiles.
        dict(name="uneven_2048", kind="uneven", scenes=2048, fp64=True, tuned=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["app", "pile", "herd", "arms", "quads", "serve", "uneven"])
    if kind == "app":
        return dict(kind=kind, bodies=_log_int(rng, 8, 128), shapes=rng.choice(["boxes", "mixed"]),
                    frames=rng.randint(1, 4))
    if kind == "pile":
        gap = rng.choice([0.02, 0.05, 0.1])
        n = _log_int(rng, 150, 700 if gap == 0.1 else 3000)
        return dict(kind=kind, bodies=n, bin=round(max(1.5, math.sqrt(n) * 0.112), 2), gap=gap, frames=1)
    if kind == "herd":
        return dict(kind=kind, quads=_log_int(rng, 8, 128), chains=rng.randint(1, 8), links=rng.randint(10, 40), frames=1)
    if kind == "arms":
        return dict(kind=kind, scenes=_log_int(rng, 1, 2048), links=rng.randint(3, 9), frames=rng.randint(1, 3))
    if kind == "quads":
        return dict(kind=kind, scenes=_log_int(rng, 4, 1024), frames=rng.randint(1, 2),
                    cone=rng.choice(["", "", "elliptic"]))
    if kind == "serve":
        n = _log_int(rng, 40, 500)
        return dict(kind=kind, scenes=n, requests=rng.randint(max(8, n // 8), n // 2))
    return dict(kind=kind, scenes=_log_int(rng, 8, 1024), fp64=rng.random() < 0.5, tuned=False)


# --- scenes ---------------------------------------------------------------------------------

SCENE_SEED = 20  # the scenes' own draws; a state's come from its seed
_SCENES = {}     # case -> what its states share: scenes built, settled and packed; tuned tiles


def _shared(case, make):
    key = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _SCENES:
        _SCENES[key] = make(case)
    return _SCENES[key]


def _random_quat(rng):
    q = rng.normal(size=4)
    return (q / np.linalg.norm(q)).tolist()


def _hull_points(rng, n):
    v = rng.normal(size=(n, 3))
    return (v / np.linalg.norm(v, axis=1, keepdims=True) * rng.uniform(0.04, 0.1, 3)).tolist()


def _app_scene(case):
    if case["shapes"] == "boxes":
        return synth.boxes_on_plane(case["bodies"], seed=SCENE_SEED)
    rng = np.random.default_rng(SCENE_SEED)
    b = SceneBuilder(fps=240, box_hulls="direct", native_hulls=True)
    b.add_ground_plane(mu=0.7)
    side = int(math.ceil(math.sqrt(case["bodies"] / 3)))
    for i in range(case["bodies"]):
        layer, cell = divmod(i, side * side)
        p = [0.3 * (cell % side), 0.3 * (cell // side), 0.15 + 0.3 * layer]
        body = b.add_body(xform=p + _random_quat(rng))
        k = i % 6
        if k == 0:
            b.add_shape_box(body, hx=0.09, hy=0.06, hz=0.07, mu=0.6)
        elif k == 1:
            b.add_shape_sphere(body, radius=0.07, mu=0.5)
        elif k == 2:
            b.add_shape_capsule(body, radius=0.04, half_height=0.07, mu=0.6)
        elif k == 3:
            b.add_shape_cylinder(body, radius=0.05, half_height=0.06, mu=0.6)
        else:
            b.add_shape_convex_hull(body, vertices=_hull_points(rng, 12 if k == 4 else 26), mu=0.6)
    return b.finalize(solver=dict(free_rigid_torsional_friction=0.02, free_rigid_rolling_friction=0.005))


def _pile_scene(case):
    """Half hulls of 8-32 points, a quarter boxes, a quarter capsules, poured into a bin of 5 boxes."""
    rng = np.random.default_rng(SCENE_SEED)
    b = SceneBuilder(fps=240, box_hulls="direct", native_hulls=True)
    opts = dict(mu=0.6, gap=case["gap"])
    half, t, h, cell = case["bin"] / 2, 0.1, 1.0, 0.25
    for pos, size in (([0, 0, -t], [half + t, half + t, t]), ([half + t / 2, 0, h / 2], [t / 2, half + t, h / 2]),
                      ([-half - t / 2, 0, h / 2], [t / 2, half + t, h / 2]), ([0, half + t / 2, h / 2], [half, t / 2, h / 2]),
                      ([0, -half - t / 2, h / 2], [half, t / 2, h / 2])):
        b.add_shape_box(-1, hx=size[0], hy=size[1], hz=size[2], xform=pos + [0, 0, 0, 1], **opts)
    row = int(case["bin"] / cell) - 1
    for i in range(case["bodies"]):
        z, k = divmod(i, row * row)
        p = [-half + cell * (1 + k % row) + rng.uniform(-0.02, 0.02),
             -half + cell * (1 + k // row) + rng.uniform(-0.02, 0.02), 0.15 + cell * z]
        body = b.add_body(xform=p + _random_quat(rng))
        kind = rng.random()
        if kind < 0.5:
            b.add_shape_convex_hull(body, vertices=_hull_points(rng, int(rng.integers(8, 33))), **opts)
        elif kind < 0.75:
            hx, hy, hz = rng.uniform(0.03, 0.1, 3).tolist()
            b.add_shape_box(body, hx=hx, hy=hy, hz=hz, **opts)
        else:
            b.add_shape_capsule(body, radius=0.02 + 0.01 * int(rng.integers(4)),
                                half_height=0.02 + 0.02 * int(rng.integers(4)), **opts)
    return b.finalize()


def _add_quadruped(b, pos, leg=0.22, **mat):
    base = b.add_body(xform=[pos[0], pos[1], pos[2], 0, 0, 0, 1])
    b.add_shape_box(base, hx=0.25, hy=0.15, hz=0.05, mass=10.0, **mat)
    for sx in (-1, 1):
        for sy in (-1, 1):
            parent, at = base, [0.2 * sx, 0.13 * sy, -0.05]
            for seg in range(3):
                link = b.add_body(xform=[pos[0] + 0.2 * sx, pos[1] + 0.13 * sy, pos[2] - 0.05 - leg * (seg + 0.5),
                                         0, 0, 0, 1])
                b.add_shape_capsule(link, radius=0.03, half_height=leg / 2 - 0.03, mass=1.2 - 0.3 * seg, **mat)
                b.add_joint_revolute(parent, link, axis=[1, 0, 0] if seg == 0 else [0, 1, 0],
                                     parent_xform=at + [0, 0, 0, 1], child_xform=[0, 0, leg / 2, 0, 0, 0, 1],
                                     targetKe=60.0, targetKd=2.0, limitLower=-1.5, limitUpper=1.5)
                parent, at = link, [0.0, 0.0, -leg / 2]


def _add_chain(b, rng, pos, links, ratio):
    parent, at = -1, list(pos)
    for k in range(links):
        mass = 0.1 * math.exp(rng.uniform(0.0, math.log(ratio)))
        body = b.add_body(xform=[pos[0], pos[1], pos[2] - 0.1 * (k + 0.5), 0, 0, 0, 1])
        b.add_shape_capsule(body, radius=0.02, half_height=0.04, mass=mass)
        b.add_joint_revolute(parent, body, axis=[0, 1, 0] if k % 2 == 0 else [1, 0, 0],
                             parent_xform=at + [0, 0, 0, 1], child_xform=[0, 0, 0.05, 0, 0, 0, 1], damping=0.05)
        parent, at = body, [0.0, 0.0, -0.05]


def _legged_scene(quads, chains, links, solver=None, **mat):
    rng = np.random.default_rng(SCENE_SEED)
    b = SceneBuilder(fps=500, box_hulls="direct", native_hulls=True)
    b.add_ground_plane(mu=0.8, **mat)
    side = max(1, int(math.ceil(math.sqrt(quads + chains))))
    for i in range(quads + chains):
        x, y = 1.2 * (i % side), 1.2 * (i // side)
        if i < quads:
            _add_quadruped(b, [x, y, 0.72], **mat)
        else:
            _add_chain(b, rng, [x, y, 0.1 * links + 0.5], links, 10.0)
    return b.finalize(solver=solver)


# The arms' links: length, capsule radius, first link's mass, the factor to the next link's, drives.
ARM = dict(length=0.3, radius=0.03, mass=2.0, ratio=0.8, ke=80.0, kd=6.0, armature=0.02, z=3.5, fps=120, substeps=4)


def _arm_axis(k):
    """Joint axes: y, x, z in turn."""
    return (1, 0, 2)[k % 3]


def _arm_scene(links):
    b = SceneBuilder(fps=ARM["fps"], box_hulls="direct", native_hulls=True)
    b.add_ground_plane(mu=0.8)
    parent, half = -1, ARM["length"] / 2
    for k in range(links):
        body = b.add_body(xform=[0, 0, ARM["z"] + ARM["length"] * (k + 0.5), 0, 0, 0, 1])
        b.add_shape_capsule(body, radius=ARM["radius"], half_height=half - 2 * ARM["radius"],
                            mass=ARM["mass"] * ARM["ratio"] ** k, gap=0.01)
        b.add_joint_revolute(parent, body, axis=[float(a == _arm_axis(k)) for a in range(3)],
                             parent_xform=[0, 0, ARM["z"] if parent < 0 else half, 0, 0, 0, 1],
                             child_xform=[0, 0, -half, 0, 0, 0, 1],
                             targetKe=ARM["ke"], targetKd=ARM["kd"], armature=ARM["armature"])
        parent = body
    return b.finalize(solver=dict(substeps=ARM["substeps"]))


def _arm_packed(case):
    scene = _arm_scene(case["links"])
    return pack(scene, caps=auto_caps(scene))


def _settled(packed, frames):
    """The packed scenes with the state that `frames` frames lead to as their initial state."""
    batch = Batch(packed)
    batch.step(frames)
    out = []
    for i, p in enumerate(packed):
        pose, vel, q, qd, _ = batch.raw_state(i)
        p = copy.copy(p)
        p.body_pose, p.body_vel, p.art = pose, vel, p.art.copy()
        p.art[p.C["A_Q"]:p.C["A_Q"] + p.NQ] = q
        p.art[p.C["A_QD"]:p.C["A_QD"] + p.ND] = qd
        out.append(p)
    batch.close()
    return out


def _moved(p, rng):
    """A scene in motion: small random velocities on its bodies and joints."""
    p = copy.copy(p)
    p.body_vel, p.art = p.body_vel.copy(), p.art.copy()
    free = np.array(p.body_kind) == 1
    v = p.body_vel.reshape(-1, 2, 4)
    v[free, 0, :3] += rng.normal(scale=0.02, size=(int(free.sum()), 3)).astype(np.float32)
    v[free, 1, :3] += rng.normal(scale=0.1, size=(int(free.sum()), 3)).astype(np.float32)
    p.art[p.C["A_QD"]:p.C["A_QD"] + p.ND] += rng.normal(scale=0.02, size=p.ND).astype(np.float32)
    return p


def _pile_packed(case):
    scene = _pile_scene(case)
    caps = auto_caps(scene)
    room = 1 << int(case["bodies"] * 32 - 1).bit_length()  # a settled pile holds more than a sparse scene
    caps.update(MAXP=2 * room, MAXC=room, MAXU=room, UH=room, WH=2 * room, AH=room)
    return _settled([pack(scene, caps=caps)], 200)


def _herd_packed(case):
    scene = _legged_scene(case["quads"], case["chains"], case["links"])
    return _settled([pack(scene, caps=auto_caps(scene))], 200)


def _quads_packed(case):
    solver, mat = None, {}
    if case["cone"]:
        solver = dict(enable_torsional_rolling_friction=True, friction_anchor_beta=0.0,
                      torsional_rolling_friction_cone=case["cone"])
        mat = dict(muTorsional=0.05, muRolling=0.01)
    scene = _legged_scene(1, 0, 0, solver, **mat)
    return _settled([pack(scene, caps=auto_caps(scene))], 200)


def _serve_packed(case):
    kinds = [(1, 0), (2, 0), (3, 0), (4, 0), (0, 1)]  # quadrupeds, chains
    scenes = [_legged_scene(q, c, 40) for q, c in kinds]
    return _settled([pack(s, caps=auto_caps(s)) for s in scenes], 200)


def _uneven_packed(case):
    opts = {"solver": {"articulation_fp64": True}} if case["fp64"] else None
    scenes = synth.uneven_batch(n_scenes=min(case["scenes"], 64), seed=SCENE_SEED)
    packed = _settled([pack(s, opts=opts, caps=auto_caps(s)) for s in scenes], 240)
    tiles = None
    if case["tuned"]:
        batch = Batch([packed[i % len(packed)] for i in range(case["scenes"])])
        tiles, _ = batch.autotune(2)
        batch.close()
    return packed, tiles


# --- the measured work ----------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng([seed, 11])
    kind = case["kind"]
    state = dict(case=case, turn=0, targets=None)
    if kind == "app":
        sim = Sim(_shared(case, _app_scene))
        sim.step(240)
        for body in range(sim.NB):
            sim.setBodyTwist(body, rng.normal(scale=[0.02] * 3 + [0.1] * 3).tolist())
        state["sim"] = sim
        return state
    spread = 0.1  # of the joint targets about the scene's own, rad
    tiles = None
    if kind == "pile":
        packed = [_moved(p, rng) for p in _shared(case, _pile_packed)]
    elif kind == "herd":
        packed = [_moved(p, rng) for p in _shared(case, _herd_packed)]
    elif kind == "arms":
        arm = _shared(case, _arm_packed)
        q, qd, state["targets"] = _arm_inputs(case, seed)
        packed = []
        for i in range(case["scenes"]):
            p = copy.copy(arm)
            p.art = arm.art.copy()
            p.art[p.C["A_Q"]:p.C["A_Q"] + p.NQ] = q[i]
            p.art[p.C["A_QD"]:p.C["A_QD"] + p.ND] = qd[i]
            packed.append(p)
    elif kind == "uneven":
        base, tiles = _shared(case, _uneven_packed)
        packed = [_moved(base[i % len(base)], rng) for i in range(case["scenes"])]
    else:
        base = _shared(case, _quads_packed if kind == "quads" else _serve_packed)
        packed = [_moved(base[i % len(base)], rng) for i in range(case["scenes"])]
    batch = Batch(packed)
    if tiles:
        batch.set_tiles(**tiles)
    joints = sum(p.ND for p in packed)
    if state["targets"] is None and joints and kind in ("herd", "quads"):
        state["targets"] = [rng.uniform(-spread, spread, joints).astype(np.float32) for _ in range(TARGET_SETS)]
    if kind == "serve":
        state["server"] = Server(batch)
        state["requests"] = [(int(rng.integers(case["scenes"])), int(rng.integers(1, 9)))
                             for _ in range(case["requests"])]
    state.update(batch=batch, poses=np.zeros(sum(8 * p.NB for p in packed), dtype=np.float32))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "app":
        state["sim"].step(case["frames"])
        return state["sim"].poses()
    batch, poses = state["batch"], state["poses"]
    if case["kind"] == "pile":
        batch.step(case["frames"])
        pose, vel, *_ = batch.raw_state(0)
        return pose, vel
    if case["kind"] == "serve":
        server, left = state["server"], case["requests"]
        for instance, frames in state["requests"]:
            server.submit(instance, frames)
        while left > 0:
            server.tick()
            left -= len(server.poll())
        batch.step_io(0, None, poses)
        return poses
    targets = None
    if state["targets"] is not None:
        targets = state["targets"][state["turn"] % len(state["targets"])]
        state["turn"] += 1
    batch.step_io(case.get("frames", 1), targets, poses)
    return poses


# Contacts per free body of a settled scene, and iterations of the solver, for the estimates below.
CONTACTS, ITERATIONS, SUBSTEPS = 3.0, 12, 4


def work(case):
    """Body and joint state and static records read once, state and poses written once per pass; the
    solver's arithmetic per contact and sweep and the articulated passes' per link and substep."""
    kind, frames = case["kind"], case.get("frames", 1)
    if kind in ("app", "pile"):
        bodies, links = case["bodies"], 0
    elif kind == "herd":
        bodies = links = 13 * case["quads"] + case["links"] * case["chains"]
    elif kind == "arms":
        bodies = links = case["scenes"] * case["links"]
    elif kind == "quads":
        bodies = links = 13 * case["scenes"]
    elif kind == "serve":  # (13 + 26 + 39 + 52 + 40) / 5 links an instance, 4.5 frames a request
        frames, bodies = 4.5, 34 * min(case["requests"], case["scenes"])
        links = bodies
    else:  # log-uniform 8-512 boxes (121 on average) and a chain of 2-40 links
        bodies, links = case["scenes"] * 142, case["scenes"] * 21
    steps = frames * SUBSTEPS
    return dict(bytes=float(bodies * (2 * 64 + 128 + 112 + 32) + links * (96 + 80 + 8 * 4)),
                flops=float(steps * (CONTACTS * (bodies - links) * (ITERATIONS * 250 + 1500)
                                     + links * (ITERATIONS * 300 + 4000))))


# --- 64-bit values --------------------------------------------------------------------------

def _arm_inputs(case, seed):
    """Joint angles and speeds, and the joint targets of TARGET_SETS control steps."""
    rng = np.random.default_rng([seed, 12])
    shape = (case["scenes"], case["links"])
    q = rng.uniform(-0.2, 0.2, shape).astype(np.float32)
    qd = rng.uniform(-0.5, 0.5, shape).astype(np.float32)
    return q, qd, [rng.uniform(-0.25, 0.25, shape).astype(np.float32).reshape(-1) for _ in range(TARGET_SETS)]


def _turn(axis, angle):
    """Rotation matrices about the unit axis `axis` (index) by `angle` [n]."""
    c, s, m = np.cos(angle), np.sin(angle), np.zeros((len(angle), 3, 3))
    i, j = (axis + 1) % 3, (axis + 2) % 3
    m[:, axis, axis] = 1.0
    m[:, i, i] = m[:, j, j] = c
    m[:, i, j], m[:, j, i] = -s, s
    return m


def _arm_frames(q):
    """Link rotations, centres and joint positions of arms with joint angles q [n, links]."""
    n, links = q.shape
    R, x = np.broadcast_to(np.eye(3), (n, 3, 3)), np.zeros((n, 3))
    x[:, 2] = ARM["z"]
    half = np.array([0.0, 0.0, ARM["length"] / 2])
    rot, com, joint = [], [], []
    for k in range(links):
        R = R @ _turn(_arm_axis(k), q[:, k])
        joint.append(x)
        rot.append(R)
        com.append(x + R @ half)
        x = x + R @ (2 * half)
    return rot, com, joint


def _capsule_inertia(r, half):
    """Principal moments of a solid capsule of unit density, and its mass."""
    L = 2 * half
    mc, ms = math.pi * r * r * L, 4 / 3 * math.pi * r ** 3
    t = mc * (L * L / 12 + r * r / 4) + ms * (0.4 * r * r + L * L / 4 + 3 * L * r / 8)
    return np.diag([t, t, 0.5 * mc * r * r + 0.4 * ms * r * r]), mc + ms


def exact(case, seed):
    """The arms' poses after the first pass: forward dynamics by the joint-space mass matrix (each
    link's centre Jacobians), Coriolis and gyroscopic terms from the link accelerations at zero joint
    acceleration, the implicit drive on the diagonal, semi-implicit Euler substeps. Scenes with
    contacts need the whole collision pipeline and have no such short computation."""
    if case["kind"] != "arms":
        return None
    q, qd, targets = _arm_inputs(case, seed)
    q, qd, target = q.astype(np.float64), qd.astype(np.float64), targets[0].astype(np.float64).reshape(q.shape)
    n, links = q.shape
    dt = 1.0 / ARM["fps"] / ARM["substeps"]
    unit, unit_mass = _capsule_inertia(ARM["radius"], ARM["length"] / 2 - 2 * ARM["radius"])
    up = np.array([0.0, 0.0, 9.81])
    for _ in range(case["frames"] * ARM["substeps"]):
        rot, com, joint = _arm_frames(q)
        axis = [rot[k][:, :, _arm_axis(k)] for k in range(links)]
        H, bias = np.zeros((n, links, links)), np.zeros((n, links))
        w = alpha = np.zeros((n, 3))
        a = np.broadcast_to(up, (n, 3))  # acceleration of the joint's point, gravity as a base acceleration
        for k in range(links):
            mass = ARM["mass"] * ARM["ratio"] ** k
            inertia = rot[k] @ (unit * (mass / unit_mass)) @ rot[k].transpose(0, 2, 1)
            alpha = alpha + np.cross(w, axis[k] * qd[:, k:k + 1])
            w = w + axis[k] * qd[:, k:k + 1]
            arm = com[k] - joint[k]
            accel = a + np.cross(alpha, arm) + np.cross(w, np.cross(w, arm))
            a = a + np.cross(alpha, 2 * arm) + np.cross(w, np.cross(w, 2 * arm))
            Jw, Jv = np.zeros((n, 3, links)), np.zeros((n, 3, links))
            for j in range(k + 1):
                Jw[:, :, j], Jv[:, :, j] = axis[j], np.cross(axis[j], com[k] - joint[j])
            H += Jw.transpose(0, 2, 1) @ inertia @ Jw + mass * Jv.transpose(0, 2, 1) @ Jv
            moment = (inertia @ alpha[:, :, None])[:, :, 0] + np.cross(w, (inertia @ w[:, :, None])[:, :, 0])
            bias += np.einsum("nij,ni->nj", Jw, moment) + mass * np.einsum("nij,ni->nj", Jv, accel)
        H += np.eye(links) * (ARM["armature"] + dt * dt * ARM["ke"] + dt * ARM["kd"])
        tau = ARM["ke"] * (target - q) - dt * ARM["ke"] * qd - ARM["kd"] * qd
        qd = qd + dt * np.linalg.solve(H, (tau - bias)[:, :, None])[:, :, 0]
        q = q + dt * qd
    out = np.zeros((n, links, 8))
    rest = np.zeros((n, 4))
    rest[:, 3] = 1.0
    _, com, _ = _arm_frames(q)
    for k in range(links):
        c, s, ax = np.cos(q[:, k] / 2), np.sin(q[:, k] / 2), _arm_axis(k)
        v, vw = rest[:, :3].copy(), rest[:, 3].copy()
        unit_axis = np.eye(3)[ax]
        rest[:, :3] = v * c[:, None] + (vw * s)[:, None] * unit_axis + s[:, None] * np.cross(v, unit_axis)
        rest[:, 3] = vw * c - s * v[:, ax]
        out[:, k, :3], out[:, k, 4:] = com[k], rest
    return out.reshape(-1)
