"""The solve's packed contact rows and its look-ahead over idle dense rows, bit for bit against the
oracle at the sizes where they can go wrong: colors with a partly filled tile, rows in shared and in
global memory, chains around the lane count and the register-held dofs, with contacts between their
links that push and contacts that do not."""
import math

import numpy as np
import pytest

from steel_webgpu_b200 import SceneBuilder, _lib, pack, synth
from steel_webgpu_b200.sim import Batch, auto_caps

pytestmark = pytest.mark.gpu

# Room for every pair of the dense scenes below (what a full buffer drops depends on the order).
ROOM = 16384
CAPS = dict(MAXP=ROOM, MAXC=ROOM, MAXU=ROOM, UH=ROOM, WH=2 * ROOM, AH=ROOM, MAXDENSE=ROOM)


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _same_as_oracle(pk, oracle_lib, frames, tiles=(), team=0):
    o = oracle_lib.OracleSim(pk)
    g = Batch([pk])
    if tiles:
        g.set_tiles(*tiles)
    if team:
        g.set_team(team)
    for _ in range(2):
        o.step(frames)
        g.step(frames)
        assert not g.stats()["overflow"]
        pose, vel, q, qd, _ = g.raw_state()
        art = o.read("art")
        assert np.array_equal(_bits(o.read("poses")[:pk.NB * 8]), _bits(pose))
        assert np.array_equal(_bits(o.read("vel")[:pk.NB * 8]), _bits(vel))
        assert np.array_equal(_bits(art[pk.C["A_Q"]:pk.C["A_Q"] + pk.NQ]), _bits(q))
        assert np.array_equal(_bits(art[pk.C["A_QD"]:pk.C["A_QD"] + pk.ND]), _bits(qd))
    stats = g.stats()
    g.close()
    return stats


def _chains(links, fold):
    """Two chains, one hanging straight, one folded by `fold` rad a joint onto itself."""
    b = SceneBuilder(fps=240)
    b.add_ground_plane(mu=0.6)
    for x, bend in ((0.0, 0.0), (2.0, fold)):
        parent, at = -1, [x, 0.0, 8.0]
        for k in range(links):
            body = b.add_body(xform=[x, 0.0, 8.0 - 0.1 * (k + 0.5), 0, 0, 0, 1])
            b.add_shape_capsule(body, radius=0.02, half_height=0.04, mass=0.2 + 0.05 * (k % 3))
            b.add_joint_revolute(parent, body, axis=[0, 1, 0], parent_xform=at + [0, 0, 0, 1],
                                 child_xform=[0, 0, 0.05, 0, 0, 0, 1], q=[bend], targetKe=2.0, targetKd=0.05)
            parent, at = body, [0.0, 0.0, -0.05]
    return b.finalize()


@pytest.mark.parametrize("links", [2, 3, 31, 32, 33, 64, 65])
def test_dense_rows(links, steel, oracle_lib):
    scene = _chains(links, 2.0)  # links two apart overlap at 2 rad a joint
    stats = _same_as_oracle(pack(scene, caps=CAPS), oracle_lib, 4)
    assert links < 3 or stats["max_dense"] > 0


@pytest.mark.parametrize("boxes", [1, 2, 7, 9, 33, 100])
@pytest.mark.parametrize("tiles", [(), (512, 4096), (32, 4096)])
def test_packed_rows(boxes, tiles, steel, oracle_lib):
    rng = np.random.default_rng(boxes)
    b = SceneBuilder(fps=240, box_hulls="direct")
    b.add_ground_plane(mu=0.6)
    side = max(1, int(math.sqrt(boxes / 3)))
    for i in range(boxes):
        layer, cell = divmod(i, side * side)
        body = b.add_body(xform=[0.21 * (cell % side), 0.21 * (cell // side), 0.101 + 0.2 * layer] + synth._rand_quat(rng)
                          if i % 5 == 4 else [0.21 * (cell % side), 0.21 * (cell // side), 0.101 + 0.2 * layer, 0, 0, 0, 1])
        b.add_shape_box(body, hx=0.1, hy=0.1, hz=0.1, mu=0.6)
    scene = b.finalize()
    _same_as_oracle(pack(scene, caps=CAPS), oracle_lib, 15, tiles)


@pytest.mark.parametrize("spin", [1e-18, 1e-21, 1e-24, 1e-30, 1e-42])
@pytest.mark.parametrize("linked", [False, True])
def test_unloaded_spin_and_rolling_rows(spin, linked, steel, oracle_lib):
    """Contacts that are near but carry no load, between bodies that turn so slowly that the square of
    the rolling impulse underflows: its length is 0, so the bound 0 does not clip it and it applies."""
    b = SceneBuilder(fps=240)
    b.add_ground_plane(mu=0.6)
    for i, (x, y, z) in enumerate(((1.0, 2.0, 0.0), (-3.0, 0.5, 4.0), (0.0, 0.0, 1.0), (-0.0, 7.0, 0.0))):
        body = b.add_body(xform=[0.5 * i, 0.0, 0.1, 0, 0, 0, 1], twist=[0.0, 0.0, 0.0, spin * x, spin * y, spin * z])
        b.add_shape_sphere(body, radius=0.08, mu=0.6)
        if linked:
            b.add_joint_free(body)
            tail = b.add_body(xform=[0.5 * i + 0.2, 0.0, 0.1, 0, 0, 0, 1])
            b.add_shape_sphere(tail, radius=0.06, mu=0.6)
            b.add_joint_revolute(body, tail, axis=[0, 1, 0], parent_xform=[0.1, 0, 0, 0, 0, 0, 1],
                                 child_xform=[-0.1, 0, 0, 0, 0, 0, 1])
    scene = b.finalize(solver=dict(free_rigid_torsional_friction=0.05, free_rigid_rolling_friction=0.01))
    _same_as_oracle(pack(scene, caps=CAPS), oracle_lib, 2)


PACKED_TILE = 15 * 128  # bytes of 8 packed rows
UNPACKED = {"coupled": ({}, {"friction_mode": "bisection"}), "momentum": (dict(nesterov_momentum=True), None),
            "compliance": (dict(contact_compliance=True, enable_restitution=False), None),
            "velocity": (dict(velocity_iterations=4), None)}


def _boxes(n, solver):
    b = SceneBuilder(fps=240, box_hulls="direct")
    b.add_ground_plane(mu=0.6)
    for i in range(n):
        body = b.add_body(xform=[0.25 * i, 0.0, 0.101, 0, 0, 0, 1])
        b.add_shape_box(body, hx=0.1, hy=0.1, hz=0.1, mu=0.6)
    return b.finalize(solver=solver)


@pytest.mark.parametrize("name", ["plain", "chain", "longest_first"] + list(UNPACKED))
def test_shared_memory_of_rows_that_are_not_there(name, steel):
    """The solve reserves shared memory for packed rows of free bodies alone, the prepare for row
    lists where the coloring makes them: what is reserved and not used is missing as L1."""
    solver, opts = UNPACKED.get(name, ({}, None))
    if name == "longest_first":
        opts = {"propagation_color_order": "longest_first"}
    scene = _chains(10, 0.0) if name == "chain" else _boxes(40, solver)
    pk = pack(scene, opts={"solver": opts} if opts else None, caps=CAPS)
    g = Batch([pk])
    solve, prep = g.layout("solve_smem"), g.layout("prep_smem")
    g.close()
    link = 268 * 4  # staged per link in both kernels; twists and impulses 64 B a body, qd 4 B a dof in the solve
    staged = link * (pk.NB if name == "chain" else 0)
    if name in ("plain", "longest_first"):
        assert solve > staged + 40 * PACKED_TILE
    else:
        assert solve <= staged + 68 * pk.NB + 1024
    if name == "longest_first":
        assert prep <= staged + 4 * 2 * pk.NB + 1024  # color counts and masks
    elif name == "plain":
        assert prep > staged + 8 * 12 * 40


@pytest.mark.parametrize("tiles", [(), (32,), (512,)])
@pytest.mark.parametrize("ext", [False, True])
def test_batch_of_packed_and_record_rows(tiles, ext, steel, oracle_lib):
    """A batch whose scenes need both solve bodies, and each scene in a batch of its own kind."""
    kinds = [({}, {"row_schedule": "contact_then_internal"} if ext else None)] + list(UNPACKED.values()) + [({}, None)]
    pks = [pack(_boxes(5 + i, solver), opts={"solver": opts} if opts else None) for i, (solver, opts) in enumerate(kinds)]
    g = Batch(pks)
    if tiles:
        g.set_tiles(*tiles)
    g.step(12)
    for i, pk in enumerate(pks):
        o = oracle_lib.OracleSim(pk)
        o.step(12)
        alone = Batch([pk])
        alone.step(12)
        for batch, scene in ((g, i), (alone, 0)):
            pose, vel = batch.raw_state(scene)[:2]
            assert np.array_equal(_bits(o.read("poses")[:pk.NB * 8]), _bits(pose)), i
            assert np.array_equal(_bits(o.read("vel")[:pk.NB * 8]), _bits(vel)), i
        alone.close()
    g.close()


@pytest.mark.parametrize("kind,count", [("flap", 1), ("flap", 17), ("flap", 33), ("floater", 2), ("floater", 5),
                                        ("floater", 33), ("quadruped", 1), ("quadruped", 3), ("quadruped", 4)])
@pytest.mark.parametrize("threads", [32, 64, 512])
def test_articulations_by_warps_and_by_threads(kind, count, threads, steel, oracle_lib):
    """Joint and impulse passes at the edges of the split: as many articulations as warps, more (by
    threads, 32 down to 1 apart), and more than threads; with contacts, limits and joint friction."""
    rng = np.random.default_rng(count)
    b = SceneBuilder(fps=240, box_hulls="direct")
    b.add_ground_plane(mu=0.6)
    for i in range(count):
        x, y = 1.2 * (i % 6), 1.2 * (i // 6)
        joint = dict(limitLower=-0.2, limitUpper=0.1, friction=0.05, velocityLimit=2.0)
        if kind == "quadruped":
            synth._add_quadruped(b, rng, [x, y, 0.7])
            continue
        base, z, at = -1, 0.05, [x - 0.1, y, 0.05]
        if kind == "floater":
            base = b.add_body(xform=[x - 0.2, y, 0.06, 0, 0, 0, 1], twist=[0.1, 0.0, 0.0, 0.0, 0.0, 1.0])
            b.add_shape_box(base, hx=0.1, hy=0.1, hz=0.05, mu=0.6)
            b.add_joint_free(base)
            at = [0.1, 0.0, -0.01]
        flap = b.add_body(xform=[x, y, z, 0, 0, 0, 1])
        b.add_shape_box(flap, hx=0.09, hy=0.1, hz=0.02, mu=0.6)
        b.add_joint_revolute(base, flap, axis=[0, 1, 0], parent_xform=at + [0, 0, 0, 1],
                             child_xform=[-0.1, 0, 0, 0, 0, 0, 1], q=[0.05 * (i % 3)], **joint)
    scene = b.finalize(solver=dict(enable_joint_friction=True, enable_joint_velocity_limits=True))
    _same_as_oracle(pack(scene, caps=CAPS), oracle_lib, 10, (threads,))


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("count", [3, 4, 7])
def test_factorisation_by_warps_and_by_threads(fp64, count, steel, oracle_lib):
    """Articulated inertias of trees with a floating base at the split's edge: three to the one warp of
    a 32-thread block, four (by threads), and both by the warps of a 512-thread block."""
    rng = np.random.default_rng(count)
    b = SceneBuilder(fps=240, box_hulls="direct")
    b.add_ground_plane(mu=0.7)
    for i in range(count):
        if i % 2 == 0:
            synth._add_quadruped(b, rng, [1.2 * i, 0.0, 0.75])
        else:
            synth._add_chain(b, rng, [1.2 * i, 0.0, 1.6], 9, ratio_max=1000.0)
    scene = b.finalize()
    pk = pack(scene, opts={"solver": {"articulation_fp64": True}} if fp64 else None, caps=CAPS)
    _same_as_oracle(pk, oracle_lib, 8, (32,))
    _same_as_oracle(pk, oracle_lib, 8, (512,))


def _sized(name):
    if name == "boxes":
        return _boxes(64, {}), None
    if name == "coupled":
        return _boxes(64, {}), {"solver": {"friction_mode": "bisection"}}
    if name == "chains":
        return _chains(40, 2.0), None
    b = SceneBuilder(fps=240, box_hulls="direct")
    b.add_ground_plane(mu=0.6)
    synth._add_quadruped(b, np.random.default_rng(1), [0.0, 0.0, 0.75])
    return b.finalize(), None


# Device bytes of a scene with its automatic capacities, alone and in a batch of 200, before rows were packed.
SCENE_BYTES = {"boxes": (1137664, 1033216), "coupled": (1109504, 1005056), "chains": (6647296, 2948608),
               "quadruped": (2587648, 1331200)}


@pytest.mark.parametrize("name", list(SCENE_BYTES))
def test_scene_bytes(name, steel):
    """Packed rows take no more device memory: batches that filled it still fit, and a byte budget of
    the serving loop admits as many instances."""
    scene, opts = _sized(name)
    pk = pack(scene, opts=opts, caps=auto_caps(scene))
    for n, limit in zip((1, 200), SCENE_BYTES[name]):
        g = Batch([pk] * n)
        assert g.scene_bytes(n - 1) <= limit
        g.close()


def _heap(boxes):
    """A plate that carries boxes: one body with more rows than a word of colors."""
    b = SceneBuilder(fps=240, box_hulls="direct")
    b.add_ground_plane(mu=0.6)
    plate = b.add_body(xform=[0.0, 0.0, 0.051, 0, 0, 0, 1])
    b.add_shape_box(plate, hx=0.7, hy=0.7, hz=0.05, mu=0.6)
    for i in range(boxes):
        body = b.add_body(xform=[0.25 * (i % 5) - 0.5, 0.25 * (i // 5) - 0.5, 0.203, 0, 0, 0, 1])
        b.add_shape_box(body, hx=0.1, hy=0.1, hz=0.1, mu=0.6)
    return b.finalize()


def _overflow_rows(g):
    """Rows of the first scene that have no color (of a table of 32), and all rows."""
    start = g.read_words("sched", g.layout("S_CSTART"), 34, dtype=np.uint32).tolist()
    return start[33] - start[32], start[33]


@pytest.mark.parametrize("boxes", [8, 9, 25])
@pytest.mark.parametrize("tiles,team", [((), 0), ((512, 4096), 0), ((32,), 0), ((), 2), ((), 5)])
def test_packed_rows_without_a_color(boxes, tiles, team, steel, oracle_lib):
    """The overflow color's rows, in global memory where the colors' are in shared memory (default
    tiles), beside them in global memory (small budget) and in a team's."""
    pk = pack(_heap(boxes), colorWords=1, caps=CAPS)
    g = Batch([pk])
    g.step(1)
    g.sync()
    over, rows = _overflow_rows(g)
    assert 0 < over < rows
    if not tiles and not team:  # the colors' rows fit what the solve has beside the bodies' twists
        assert g.layout("solve_smem") > 64 * pk.NB + PACKED_TILE * (rows // 8 + 1)
    g.close()
    _same_as_oracle(pk, oracle_lib, 6, tiles, team)


def test_coloring_wait_that_runs_out(steel, oracle_lib):
    """One pass a thread is not enough for a body's rows: the step reports the timeout, with the rows left
    in the overflow color; with the default limit back, a reset replays the scene bit for bit."""
    pk = pack(_heap(8), colorWords=1, caps=CAPS)  # its lists fit shared memory: 12 rows a body
    g = Batch([pk])
    g.step(1)
    g.sync()
    colored = _overflow_rows(g)
    g.reset()
    _lib.check(_lib.load().steel_debug_set_wait_limit(g.h, 4))
    g.step(1)
    with pytest.raises(_lib.SteelError, match="coloring") as e:
        g.sync()
    assert e.value.code == 7
    over, rows = _overflow_rows(g)
    assert rows == colored[1] and over > colored[0]
    assert np.isfinite(g.poses()).all()
    _lib.check(_lib.load().steel_debug_set_wait_limit(g.h, 16777216))
    g.reset()
    o = oracle_lib.OracleSim(pk)
    g.step(6)
    o.step(6)
    assert np.array_equal(_bits(o.read("poses")[:pk.NB * 8]), _bits(g.poses()))
    g.close()


@pytest.mark.parametrize("what", ["parent", "parent_nan", "range"])
def test_links_out_of_range_are_refused(what, steel):
    """The levels of the articulation trees are built on the host from the packed records: a parent or a
    range of links that the scene does not have is an error there."""
    pk = pack(_chains(3, 0.0), caps=CAPS)
    if what == "range":
        pk.statU = pk.statU.copy()
        pk.statU[pk.C["SU_ART"] + 1] = pk.C["NL"] + 1
    else:
        pk.statF = pk.statF.copy()
        pk.statF.reshape(-1, 4)[pk.C["SF_LINK"] + 6, 1] = np.nan if what == "parent_nan" else pk.C["NL"]
    with pytest.raises(_lib.SteelError) as e:
        Batch([pk])
    assert e.value.code == 1
