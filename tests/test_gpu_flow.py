"""The chunked PGS kernel at the edges of its deal, against the team kernel, bit for bit.

Both solve the groups in (sweep, colour, pair) order, so every state must be identical: a warp with
one item a sweep (few groups a chunk), several rounds of a colour, groups of 1 to 4 rows in one
warp, split groups of a deep initial overlap, kinematic bodies, no velocity sweep and a single one.
BGPU_PGS=team selects the team kernel (read once per process), hence the child processes.
"""
import os
import subprocess
import sys
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import time
sys.path[:0] = [sys.argv[1] + "/bullet-physics_b200"]
import numpy as np
import bgpu, scenes
kind, iters, steps = sys.argv[2], int(sys.argv[3]), int(sys.argv[4])
if kind == "boxes":        # 1,050 bodies: the smallest worlds cut into chunks, a few groups a chunk
    s = scenes.falling_box_stack(7, 6, 25, seed=9)
elif kind == "mixed":      # every row count, deep overlaps at the start (split groups, many colours)
    s = scenes.mixed_convex_pile(1500, seed=8, extent=9.0)
else:                      # several rounds of the large colours per warp
    s = scenes.large_pile_fast(40, 40, 14, seed=7, spacing=1.0)
s.iterations = iters
w = s.build_gpu(bgpu)
if kind == "boxes":        # a kinematic body in the stack's way
    w.add_body(1, (0.0, 1.0, 0.0), linvel=(0.3, 0.0, 0.0), mass=0.0, kinematic=1)
out = []
for _ in range(steps):
    w.step(s.dt)
    out.append(w.state())
assert w.stats()["device_status"] == 0
np.save(sys.argv[5], np.stack(out))
"""


@pytest.mark.parametrize("kind,iters,steps", [("boxes", 10, 70), ("boxes", 0, 40), ("boxes", 1, 60),
                                              ("mixed", 10, 30), ("pile", 7, 25)])
def test_chunked_kernel_equals_team_kernel(tmp_path, kind, iters, steps):
    states = []
    for mode in ("", "team"):
        env = dict(os.environ)
        env.pop("BGPU_PGS", None)
        if mode:
            env["BGPU_PGS"] = mode
        out = str(tmp_path / f"s{mode}.npy")
        r = subprocess.run([sys.executable, "-c", CHILD, ROOT, kind, str(iters), str(steps), out], env=env,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-1500:]
        states.append(np.load(out))
    np.testing.assert_array_equal(*states)


@pytest.mark.parametrize("n", [255, 256, 1024, 1025])
def test_plain_worlds_on_both_sides_of_the_lines(gpu_oracle, n):
    """One block (up to 255 bodies), one block to prepare and many to solve (256 to 1,024), chunks
    (more): each step equals the oracle's from the same state."""
    bgpu, orc, scenes = gpu_oracle
    s = scenes.large_pile(nx=6, nz=6, ny=-(-(n - 1) // 36), seed=n, spacing=1.0)
    for f in ("shape_of", "pos", "quat", "linvel", "angvel", "mass", "friction", "restitution"):
        setattr(s, f, getattr(s, f)[:n])
    g, o = s.build_gpu(bgpu), s.build_oracle(orc)
    for _ in range(12):
        g.step(s.dt)
        o.set_solve_order(g.solve_order())
        o.step(s.dt)
        a, b = g.state(), o.state()
        assert np.abs(a[:, :13] - b[:, :13]).max() <= 1e-5 * max(1.0, np.abs(b[:, :13]).max())
    assert g.num_bodies == n and g.stats()["num_contacts"] > n and g.stats()["device_status"] == 0


def _plain_and_one_block(bgpu, s, kinematic):
    """The scene as a plain world and as a batch of one world, which one block solves."""
    a = s.arrays()
    d = bgpu.desc_array(a["shape"], a["pos"], a["quat"], a["linvel"], a["angvel"], a["mass"], a["friction"],
                        a["restitution"])
    if kinematic:
        d["mass"][-1], d["flags"][-1], d["linear_velocity"][-1] = 0.0, bgpu.KINEMATIC, (0.5, 0.0, 0.0)
    out = []
    for batch in (False, True):
        w = bgpu.World(gravity=s.gravity, batch=batch, num_iterations=s.iterations)
        import scenes
        scenes.add_shapes(w, s.shapes)
        first, n = bgpu.ctypes.c_uint32(), bgpu.ctypes.c_uint32(len(d))
        p = d.ctypes.data_as(bgpu.ctypes.POINTER(bgpu.BodyDesc))
        if batch:
            bgpu.check(w.L.bgpu_batch_add_worlds(w.h, 1, bgpu.ctypes.byref(n), p, bgpu.ctypes.byref(first)), "add_worlds")
            w.set_tuning(256, 0)
        else:
            bgpu.check(w.L.bgpu_add_bodies(w.h, len(d), p, bgpu.ctypes.byref(first)), "add_bodies")
        out.append(w)
    return out


@pytest.mark.parametrize("kind,iters", [("boxes", 10), ("boxes", 0), ("boxes", 1), ("mixed", 0), ("mixed", 1),
                                        ("mixed", 10), ("pile", 25)])
def test_many_blocks_equal_one(gpu_oracle, kind, iters):
    """Worlds of 256 to 1,024 bodies, solved by many blocks, against one block, bit for bit: a kinematic body,
    deep overlaps (split groups), groups of every row count, no velocity sweep, one and many."""
    bgpu, _, scenes = gpu_oracle
    s = {"boxes": lambda: scenes.falling_box_stack(7, 6, 7, seed=9),
         "mixed": lambda: scenes.mixed_convex_pile(700, seed=8, extent=7.0),
         "pile": lambda: scenes.large_pile(10, 10, 10, seed=7, spacing=1.0)}[kind]()
    s.iterations = iters
    plain, one = _plain_and_one_block(bgpu, s, kind == "boxes")
    assert 256 <= plain.num_bodies <= 1024
    split = 0
    for step in range(60 if kind == "boxes" else 30):
        plain.step(s.dt)
        one.step(s.dt)
        np.testing.assert_array_equal(plain.state(), one.state(), err_msg=f"step {step}")
        split += plain.stats()["num_split_pairs"]
    assert plain.stats()["num_contacts"] > 0 and (kind != "mixed" or split > 0)


@pytest.mark.parametrize("n", [200, 300, 1000])
def test_gradients_of_a_plain_world(gpu_oracle, n):
    """A tape over a plain world (one block up to 255 bodies, many beyond) against the same world as a batch of one.
    The reverse pass adds up a body's terms in its colours' order either way; only the friction and
    restitution gradients add theirs by atomics, whose order is free: 1e-5 of the largest."""
    bgpu, _, scenes = gpu_oracle
    s = scenes.large_pile(nx=6, nz=6, ny=-(-n // 36), seed=n, spacing=1.0)
    for f in ("shape_of", "pos", "quat", "linvel", "angvel", "mass", "friction", "restitution"):
        setattr(s, f, getattr(s, f)[:n])
    grads = []
    for w in _plain_and_one_block(bgpu, s, False):
        w.step(s.dt, 20)
        t = bgpu.Tape(w, 6)
        t.forward(s.dt, 15)
        gx = np.random.default_rng(n).normal(size=(n, 3)).astype(np.float32)
        grads.append(t.backward(gx))
        assert w.stats()["num_contacts"] > n // 2
    for k in ("v0", "w0", "friction", "restitution"):
        scale = np.abs(grads[1][k]).max()
        np.testing.assert_allclose(grads[0][k], grads[1][k], rtol=0.0, atol=1e-5 * max(scale, 1e-30), err_msg=k)
    assert np.abs(grads[1]["v0"]).max() > 0.0 and np.abs(grads[1]["friction"]).max() > 0.0


@pytest.fixture(scope="module")
def gpu_oracle():
    sys.path[:0] = [os.path.join(ROOT, "bullet-physics_b200"), os.path.join(ROOT, "tests")]
    import bgpu
    import oracle_api
    import scenes
    return bgpu, oracle_api, scenes


def test_worlds_of_different_sizes_step_side_by_side(gpu_oracle):
    """The shared-memory limit of the per-world kernel is the process's: a later, smaller world must
    not lower it for an earlier one."""
    bgpu, _, scenes = gpu_oracle
    big = scenes.batched_worlds(4, seed=1, min_bodies=200, max_bodies=220).build_gpu(bgpu)
    big.set_tuning(256, 0x7fffffff)
    small = scenes.batched_worlds(4, seed=1, min_bodies=8, max_bodies=9).build_gpu(bgpu)
    for w in (big, small, big):
        w.step(1.0 / 60.0, 30)
        assert w.stats()["device_status"] == 0


@pytest.mark.parametrize("balls,layers,iters", [(70, 3, 10), (70, 3, 0), (140, 11, 20)])
def test_a_body_with_more_neighbours_than_colours(gpu_oracle, balls, layers, iters):
    """A heavy tray with more balls on it than a colouring has colours (64 and 128), one in three of them sunk
    deep enough for a split row, no gravity: the step reports the overflow and nothing else, at once, every
    group is still solved (the balls stop, the sunk ones are pushed out), and a pile beside the tray
    moves as it does without it, bit for bit."""
    bgpu, _, scenes = gpu_oracle
    is_box, ppos, pquat = scenes.large_pile_arrays(10, 10, layers, 4, 1.0)
    ppos = ppos + np.array([40.0, 0.0, 0.0])
    pile = len(ppos)
    k = np.arange(balls)
    sunk = k % 3 == 0
    bpos = np.stack([(k % 12) * 0.5 - 2.75, np.where(sunk, 5.395, 5.445), (k // 12) * 0.5 - 2.75], axis=1)

    def world(tray):
        w = bgpu.World(gravity=(0.0, 0.0, 0.0), num_iterations=iters)
        plane, box, sph = w.plane([0.0, 1.0, 0.0], 0.0), w.box([0.5, 0.5, 0.5]), w.sphere(0.5)
        shape = np.concatenate([[plane], np.where(is_box, box, sph)])
        pos, quat = np.concatenate([np.zeros((1, 3)), ppos]), np.concatenate([[[0, 0, 0, 1]], pquat])
        mass = np.concatenate([[0.0], np.ones(pile)])
        vel = np.zeros((1 + pile, 3))
        if tray:
            shape = np.concatenate([shape, [w.box([4.0, 0.25, 4.0])], np.full(balls, w.sphere(0.2))])
            pos = np.concatenate([pos, [[0.0, 5.0, 0.0]], bpos])
            quat = np.concatenate([quat, np.tile([0, 0, 0, 1], (balls + 1, 1))])
            mass = np.concatenate([mass, [1e5], np.ones(balls)])
            vel = np.concatenate([vel, np.zeros((1, 3)), np.tile([0.0, -0.1, 0.0], (balls, 1))])
        w.add_bodies_array(shape, pos, quat, linvel=vel, mass=mass)
        return w

    w, alone = world(True), world(False)
    for step in range(3):
        alone.step(1.0 / 60.0)
        t0 = time.perf_counter()
        with pytest.raises(bgpu.BgpuError, match="device status bits 0x8$"):
            w.step(1.0 / 60.0)
        assert step == 0 or time.perf_counter() - t0 < 1.0
        assert w.stats()["device_status"] == 8 and w.stats()["num_contact_pairs"] >= balls
        np.testing.assert_array_equal(w.state()[:pile + 1], alone.state())
    assert alone.stats()["num_contacts"] > 0
    ball = w.state()[pile + 2:]
    if iters:  # (without a sweep there are no impulses)
        assert (ball[:, 8] > -0.02).all() and (ball[:, 1] > bpos[:, 1] - 2e-3).all()
        assert (ball[sunk, 1] > bpos[sunk, 1] + 1e-3).all()
