"""The workloads the library's speed is measured on, through its public entry points.

Every case builds one world (or one batch of worlds) with the recipes of
`bullet-physics_b200/scenes.py`, lets it settle for a number of steps, and then
times what a caller does with it: step it and read the poses or the states
back. `listed()` names the fixed cases, `draw()` makes more of the same kinds
over the same ranges.

A case's `kind`:
  frames    a game or teaching scene: forces up (optional), one step, poses or states down; the world
            goes on from pass to pass and its bodies never sleep, so each pass has contacts to solve
  rollout   a planner's rollout: back to a checkpoint, a number of steps, poses down
  adjoint   one iteration of an optimiser over a rollout: forward, gradients, back to the start
"""
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bullet-physics_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import bgpu  # noqa: E402
import scenes  # noqa: E402

AWAKE = scenes.ACT_DISABLE_DEACTIVATION
DT = 1.0 / 60.0


def listed():
    return [
        # The smallest call there is: eight stacked boxes, one frame. Launches and latency only.
        dict(name="tiny_frame", kind="frames", scene="boxes", nx=2, ny=2, nz=2, settle=90, forces=False, steps=1),
        # The 1,000-box stack of the benchmark: a rollout while its layers rest on each other.
        dict(name="stack_1000", kind="rollout", scene="boxes", nx=10, ny=10, nz=10, settle=80, steps=10),
        # The terrain scene rain_500: boxes, spheres and capsules on a triangle mesh.
        dict(name="rain_500", kind="rollout", scene="terrain", nx=10, nz=10, layers=5, grid=20, settle=90, steps=10),
        # The joint scene: 150 chains of three boxes on spring-2 joints; one frame, states down.
        dict(name="chains_150", kind="frames", scene="chains", count=150, links=3, settle=10, forces=False, steps=1),
        # An interactive frame of a mid-size pile of ragged size: forces up, one step, states down.
        dict(name="pile_frame_5681", kind="frames", scene="pile", nx=23, ny=13, nz=19, settle=90, forces=True, steps=1),
        # Many bodies that fly by each other: broad phase, narrow phase without a hit, integration.
        dict(name="sparse_60000", kind="rollout", scene="sparse", n=60000, settle=0, steps=4),
        # The 16,384-body mixed convex pile: every narrow-phase route, GJK/EPA among them.
        dict(name="mixed_16384", kind="rollout", scene="mixed", n=16384, extent=40, settle=100, steps=8),
        # The headline: the pile of 131,072 boxes and spheres, 20 iterations.
        dict(name="pile_131072", kind="rollout", scene="pile", nx=64, ny=32, nz=64, settle=100, steps=8),
        # The batched worlds of the benchmark (about 288,000 bodies), with the launch shape that the
        # autotuner settles on for them (128 threads, worlds of up to 128 bodies one per warp).
        dict(name="worlds_4096", kind="rollout", scene="worlds", n=4096, lo=8, hi=256, settle=60, steps=8, tune=True),
        # A small batch of a few dozen environments, launch shape as it comes.
        dict(name="worlds_96", kind="rollout", scene="worlds", n=96, lo=8, hi=256, settle=60, steps=8, tune=False),
        # The adjoint worlds of the benchmark: 1,024 worlds of 64 boxes, forward and backward.
        dict(name="adjoint_1024", kind="adjoint", scene="throw", n=1024, side=4, steps=40, every=20),
        # Fast bodies with swept-sphere clamps raining onto thin plates.
        dict(name="ccd_rain_2048", kind="rollout", scene="ccd", fast=2048, boxes=1024, plates=16, settle=2, steps=4),
    ]


def _log(rng, lo, hi):
    """A whole number, its logarithm spread evenly over [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    which = rng.choice(["tiny", "stack", "rain", "chains", "frame", "sparse", "mixed", "pile", "worlds", "adjoint",
                        "ccd"])
    if which == "tiny":
        return dict(kind="frames", scene="boxes", nx=rng.randint(1, 4), ny=rng.randint(1, 4), nz=rng.randint(1, 4),
                    settle=rng.randint(60, 120), forces=rng.random() < 0.5, steps=rng.randint(1, 2))
    if which == "stack":
        return dict(kind="rollout", scene="boxes", nx=rng.randint(3, 10), ny=rng.randint(3, 10),
                    nz=rng.randint(3, 10), settle=rng.randint(40, 120), steps=rng.randint(4, 10))
    if which == "rain":
        g = rng.randint(5, 20)
        return dict(kind="rollout", scene="terrain", nx=g, nz=rng.randint(5, 20), layers=rng.randint(2, 5),
                    grid=2 * g, settle=rng.randint(60, 120), steps=rng.randint(2, 10))
    if which == "chains":
        return dict(kind="frames", scene="chains", count=_log(rng, 5, 5000), links=rng.randint(1, 4),
                    settle=rng.randint(5, 20), forces=rng.random() < 0.5, steps=1)
    if which == "frame":
        return dict(kind="frames", scene="pile", nx=rng.randint(6, 40), ny=rng.randint(4, 20), nz=rng.randint(6, 40),
                    settle=rng.randint(60, 120), forces=True, steps=1)
    if which == "sparse":
        return dict(kind="rollout", scene="sparse", n=_log(rng, 500, 60000), settle=0, steps=rng.randint(2, 4))
    if which == "mixed":
        n = _log(rng, 300, 16384)
        return dict(kind="rollout", scene="mixed", n=n, extent=max(8, int(round(40.0 * (n / 16384.0) ** (1.0 / 3.0)))),
                    settle=rng.randint(60, 120), steps=rng.randint(2, 8))
    if which == "pile":
        return dict(kind="rollout", scene="pile", nx=_log(rng, 9, 64), ny=rng.randint(6, 32), nz=_log(rng, 9, 64),
                    settle=rng.randint(60, 120), steps=rng.randint(2, 8))
    if which == "worlds":
        n = _log(rng, 8, 4096)
        return dict(kind="rollout", scene="worlds", n=n, lo=8, hi=rng.choice([64, 256]), settle=rng.randint(30, 60),
                    steps=rng.randint(2, 8), tune=n >= 1024)
    if which == "adjoint":
        return dict(kind="adjoint", scene="throw", n=_log(rng, 8, 1024), side=rng.randint(2, 4),
                    steps=rng.randint(10, 40), every=rng.choice([10, 20]))
    return dict(kind="rollout", scene="ccd", fast=_log(rng, 16, 2048), boxes=_log(rng, 32, 1024),
                plates=rng.randint(4, 16), settle=rng.randint(0, 3), steps=rng.randint(2, 4))


# ---------------------------------------------------------------- worlds
def _add(w, shape, pos, quat=None, linvel=None, angvel=None, mass=None, friction=None, restitution=None, awake=False):
    """Bodies from arrays; awake: the dynamic ones never sleep."""
    n = len(shape)
    if quat is None:
        quat = np.tile(np.array([0, 0, 0, 1], np.float32), (n, 1))
    d = bgpu.desc_array(shape, pos, quat, linvel, angvel, mass, friction, restitution)
    if awake:
        d["activation"] = np.where(d["mass"] > 0, AWAKE, 0).astype(np.uint32)
    first = bgpu.ctypes.c_uint32()
    bgpu.check(w.L.bgpu_add_bodies(w.h, n, d.ctypes.data_as(bgpu.ctypes.POINTER(bgpu.BodyDesc)),
                                   bgpu.ctypes.byref(first)), "add_bodies")


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    return (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)


def _scene_world(s, awake):
    w = bgpu.World(gravity=s.gravity, num_iterations=s.iterations)
    scenes.add_shapes(w, s.shapes)
    a = s.arrays()
    _add(w, a["shape"], a["pos"], a["quat"], a["linvel"], a["angvel"], a["mass"], a["friction"], a["restitution"], awake)
    return w


def _terrain(case, seed):
    """mesh_rain's lattice over its wavy terrain, each body a little off its lattice point."""
    s = scenes.mesh_rain(case["nx"], case["nz"], case["layers"], case["grid"])
    rng = np.random.default_rng(seed)
    pos = np.asarray(s.pos, dtype=np.float32)
    pos[1:] += rng.uniform(-0.1, 0.1, size=(len(pos) - 1, 3)).astype(np.float32)
    s.pos = list(pos)
    return s


def _pile_world(case, seed, awake):
    is_box, pos, quat = scenes.large_pile_arrays(case["nx"], case["nz"], case["ny"], seed)
    w = bgpu.World(num_iterations=20)
    plane = w.plane([0.0, 1.0, 0.0], 0.0)
    box, sph = w.box([0.5, 0.5, 0.5]), w.sphere(0.5)
    n = len(pos)
    _add(w, np.concatenate([[plane], np.where(is_box, box, sph)]), np.concatenate([np.zeros((1, 3)), pos]),
         np.concatenate([[[0, 0, 0, 1]], quat]), mass=np.concatenate([[0.0], np.ones(n)]), awake=awake)
    return w


def _mixed_world(case, seed):
    """mixed_convex_pile's kinds and sizes; the bodies share a few dozen shapes of each kind, and a
    hull's mass is that of its ball times 0.7 (a 24-point hull's share of it)."""
    rng = np.random.default_rng(seed)
    n, e = case["n"], float(case["extent"])
    w = bgpu.World(num_iterations=10)
    plane = w.plane([0.0, 1.0, 0.0], 0.0)
    ids, masses = [], []
    pools = []
    for kind, size in enumerate((64, 48, 24, 24)):
        pool = []
        for _ in range(size):
            if kind == 0:
                h = rng.uniform(0.2, 0.6, size=3)
                sh, m = w.box(h), 8000.0 * h.prod()
            elif kind == 1:
                r = rng.uniform(0.2, 0.5)
                sh, m = w.sphere(r), 4000.0 / 3.0 * np.pi * r ** 3
            elif kind == 2:
                r, hh = rng.uniform(0.1, 0.3), rng.uniform(0.2, 0.6)
                sh, m = w.capsule(r, hh), 1000.0 * (np.pi * r * r * 2.0 * hh + 4.0 / 3.0 * np.pi * r ** 3)
            else:
                r = rng.uniform(0.3, 0.6)
                sh, m = w.hull(scenes.fibonacci_free_points(rng, 24, r)), 700.0 * 4.0 / 3.0 * np.pi * r ** 3
            pool.append(len(ids))
            ids.append(sh)
            masses.append(m)
        pools.append(np.asarray(pool))
    kinds = rng.choice(4, size=n, p=[0.4, 0.3, 0.15, 0.15])
    pick = rng.random(n)
    which = np.empty(n, dtype=np.int64)
    for k in range(4):
        at = kinds == k
        which[at] = pools[k][(pick[at] * len(pools[k])).astype(np.int64)]
    ids, masses = np.asarray(ids), np.asarray(masses)
    pos = np.stack([rng.uniform(-e / 2, e / 2, n), rng.uniform(1.0, 1.0 + e, n), rng.uniform(-e / 2, e / 2, n)], axis=1)
    _add(w, np.concatenate([[plane], ids[which]]), np.concatenate([np.zeros((1, 3)), pos]),
         np.concatenate([[[0, 0, 0, 1]], _rotations(rng, n)]), mass=np.concatenate([[0.0], masses[which]]))
    return w


def _sparse(case, seed):
    """Spheres (r 0.5) and cubes (half 0.3) near the points of a face-centred lattice, 1.27 m apart:
    neighbours' boxes overlap, the bodies themselves stay clear of each other over the case's steps.
    No gravity, a little damping, forces and torques for the first step."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    cells = int(np.ceil((n / 4.0) ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), axis=-1).reshape(-1, 1, 3)
    base = (g + np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])).reshape(-1, 3)[:n] * 1.8
    f32 = np.float32
    return dict(cube=rng.random(n) < 0.4, pos=(base + rng.uniform(-0.03, 0.03, (n, 3))).astype(f32),
                quat=_rotations(rng, n), linvel=rng.uniform(-0.4, 0.4, (n, 3)).astype(f32),
                angvel=rng.uniform(-2.0, 2.0, (n, 3)).astype(f32), mass=rng.uniform(0.8, 1.2, n).astype(f32),
                force=rng.uniform(-4.0, 4.0, (n, 3)).astype(f32), torque=rng.uniform(-1.0, 1.0, (n, 3)).astype(f32))


SPARSE_DAMPING = 0.1


def _sparse_world(a):
    w = bgpu.World(gravity=(0.0, 0.0, 0.0), num_iterations=10)
    sph, box = w.sphere(0.5), w.box([0.3, 0.3, 0.3])
    n = len(a["pos"])
    d = bgpu.desc_array(np.where(a["cube"], box, sph), a["pos"], a["quat"], a["linvel"], a["angvel"], a["mass"])
    d["linear_damping"] = d["angular_damping"] = SPARSE_DAMPING
    first = bgpu.ctypes.c_uint32()
    bgpu.check(w.L.bgpu_add_bodies(w.h, n, d.ctypes.data_as(bgpu.ctypes.POINTER(bgpu.BodyDesc)),
                                   bgpu.ctypes.byref(first)), "add_bodies")
    return w


def _batch_world(case, seed):
    """batched_worlds with its world sizes as the recipe deals them, every body nudged sideways."""
    s = scenes.batched_worlds(case["n"], 4, min_bodies=case["lo"], max_bodies=case["hi"])
    rng = np.random.default_rng(seed)
    for world in s.worlds:
        n = len(world["pos"]) - 1
        world["pos"][1:, 0::2] += rng.uniform(-0.02, 0.02, (n, 2)).astype(np.float32)
    return s.build_gpu(bgpu)


# ---------------------------------------------------------------- the measured passes
def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


def prepare(case, seed):
    scene, awake, dt = case["scene"], case["kind"] == "frames", DT
    rng = np.random.default_rng(seed)
    s = {"case": case}
    if scene == "boxes":
        w = _scene_world(scenes.falling_box_stack(case["nx"], case["ny"], case["nz"], seed), awake)
    elif scene == "terrain":
        w = _scene_world(_terrain(case, seed), awake)
    elif scene == "chains":
        w = scenes.spring2_chains_world(bgpu, case["count"], links=case["links"])
        st = w.state()  # each chain starts with a push of its own
        st[:, 7:10] += np.where(st[:, 13:14] == AWAKE, rng.uniform(-1.0, 1.0, (len(st), 3)), 0.0)
        w.set_state(st)
    elif scene == "pile":
        w = _pile_world(case, seed, awake)
    elif scene == "sparse":
        a = _sparse(case, seed)
        w = _sparse_world(a)
        s["force"], s["torque"] = a["force"], a["torque"]
    elif scene == "mixed":
        w = _mixed_world(case, seed)
    elif scene == "worlds":
        w = _batch_world(case, seed)
    elif scene == "throw":
        dt = 1.0 / 120.0
        w = scenes.adjoint_worlds(case["n"], seed, side=case["side"]).build_gpu(bgpu)
    elif scene == "ccd":
        w, _ = scenes.ccd_rain_world(bgpu, case["fast"], case["boxes"], case["plates"], seed)
    else:
        raise ValueError(scene)
    n = w.num_bodies
    if case.get("settle"):
        w.step(dt, case["settle"])
    s["world"], s["dt"] = w, dt
    if case["kind"] == "frames":
        # A state in these ranges is small: the caller reads all of it (velocities, activation).
        s["force"] = None
        if case["forces"]:
            s["force"] = rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)
            s["torque"] = rng.uniform(-0.2, 0.2, (n, 3)).astype(np.float32)
        return s
    s["poses"] = _pinned(n, 7)
    if scene == "ccd":  # a tape does not cover the clamps: these rollouts start from a state kept on the host
        s["start"] = w.state()
        return s
    if case["kind"] == "adjoint":
        s["goal"] = (w.state()[:, 0:3] + np.array([1.0, 0.0, 0.5])).astype(np.float32)
        s["tape"] = bgpu.Tape(w, case["every"])
        s["tape"].forward(dt, case["steps"])
        return s
    if case.get("tune"):
        w.set_tuning(128, 128)
    s["tape"] = bgpu.Tape(w, 1)
    s["tape"].forward(dt, 1)  # its first checkpoint is the state the rollouts start from
    return s


def run(s):
    case, w = s["case"], s["world"]
    if case["kind"] == "frames":
        if s["force"] is not None:
            w.apply_forces(s["force"], s["torque"])
        w.step(s["dt"], case["steps"])
        return w.state()
    if "start" in s:
        w.set_state(s["start"])
    else:
        s["tape"].rewind()
    if case["kind"] == "adjoint":
        s["tape"].forward(s["dt"], case["steps"])
        poses = w.poses(s["poses"])
        grads = s["tape"].backward(2.0 * (poses[:, 0:3] - s["goal"]))
        return [poses, grads["v0"], grads["w0"], grads["friction"], grads["restitution"]]
    if s.get("force") is not None:
        w.apply_forces(s["force"], s["torque"])
    w.step(s["dt"], case["steps"])
    return w.poses(s["poses"])


# ---------------------------------------------------------------- what a pass cannot do without
# Bodies, contacts per body and joint rows of the settled scenes (contacts: as bgpu_get_stats reports them).
_CONTACTS = {"boxes": 4.0, "terrain": 2.0, "chains": 0.0, "pile": 3.8, "sparse": 0.0, "mixed": 2.0, "worlds": 2.5,
             "throw": 2.0, "ccd": 0.5}


def _bodies(case):
    scene = case["scene"]
    if scene in ("boxes", "pile"):
        return case["nx"] * case["ny"] * case["nz"]
    if scene == "terrain":
        return case["nx"] * case["nz"] * case["layers"]
    if scene == "chains":
        return case["count"] * (case["links"] + 1)
    if scene == "worlds":  # mean of exp(U(ln lo, ln hi))
        return case["n"] * (case["hi"] - case["lo"]) / np.log(case["hi"] / case["lo"])
    if scene == "throw":
        return case["n"] * case["side"] ** 3
    if scene == "ccd":
        return case["fast"] + case["boxes"] + case["plates"] ** 2
    return case["n"]


def work(case):
    """Bytes: each body's pose and velocities and each contact's manifold point (80 bytes) read and
    written once a pass. Operations: about 250 for a contact or joint row group and sweep (three
    sweeps' worth backward, which replays and reverses each step), 1,000 a body and step."""
    n = float(_bodies(case))
    contacts = n * _CONTACTS[case["scene"]]
    rows = contacts + (case["count"] * case["links"] * 3.0 if case["scene"] == "chains" else 0.0)
    iters = 20.0 if case["scene"] == "pile" else 10.0
    passes = 3.0 if case["kind"] == "adjoint" else 1.0
    return {"bytes": 2.0 * (52.0 * n + 80.0 * contacts),
            "flops": passes * case["steps"] * (rows * (iters + 1.0) * 250.0 + 1000.0 * n)}


# ---------------------------------------------------------------- 64 bits
def exact(case, seed):
    """The sparse scene in closed form, step by step: no body touches another. The other scenes have
    contacts or joints: a step's sequential solve depends on the order of its rows, and its contact
    set on f32 decisions, so a 64-bit step is another trajectory and not a value of this one."""
    if case["scene"] != "sparse":
        return None
    a = _sparse(case, seed)
    f64 = np.float64
    dt = f64(np.float32(DT))
    x, q, v, w, m = (a[k].astype(f64) for k in ("pos", "quat", "linvel", "angvel", "mass"))
    half = f64(np.float32(0.3))
    inertia = np.where(a["cube"], m / 3.0 * 2.0 * half * half, 0.4 * m * 0.25)  # a multiple of the identity
    keep = (1.0 - f64(np.float32(SPARSE_DAMPING))) ** dt
    for step in range(case["steps"]):
        v, w = v * keep, w * keep
        if step == 0:  # the forces of a call act in its first step
            v = v + a["force"].astype(f64) / m[:, None] * dt
            w = w + a["torque"].astype(f64) / inertia[:, None] * dt
        x = x + v * dt
        speed = np.linalg.norm(w, axis=1)
        axis = w * (np.sin(0.5 * speed * dt) / speed)[:, None]
        s = np.cos(0.5 * speed * dt)
        qv, qs = q[:, 0:3], q[:, 3]
        q = np.concatenate([s[:, None] * qv + qs[:, None] * axis + np.cross(axis, qv),
                            (s * qs - (axis * qv).sum(axis=1))[:, None]], axis=1)
        q = q / np.linalg.norm(q, axis=1, keepdims=True)
    return np.concatenate([x, q], axis=1)
