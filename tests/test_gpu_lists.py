"""The ordered lists of a step at the edges of their tiles (256 and 1,024 pairs, 4,096 from 256k pairs
on) and the manifold cache with and without pruning, against the oracle step by step."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path[:0] = [os.path.join(ROOT, "bullet-physics_b200"), os.path.join(ROOT, "tests")]


@pytest.mark.parametrize("npairs", [1, 255, 256, 257, 1023, 1024, 1025, 5000])
def test_contact_lists_at_tile_edges(npairs):
    """npairs separate pairs of touching spheres, with and without a gap of pairs that only overlap."""
    import bgpu
    import oracle_api as orc

    g, o = bgpu.World(num_iterations=4), orc.OracleWorld("f32")
    o.set_gravity((0.0, -9.81, 0.0))
    o.set_solver(num_iterations=4)
    side = int(np.ceil(npairs ** 0.5))
    k = np.arange(npairs)
    base = np.stack([(k % side) * 4.0, np.zeros(npairs), (k // side) * 4.0], axis=1)
    gap = np.where(k % 3 == 1, 1.03, 0.98)  # every third pair: boxes overlap, spheres do not touch
    pos = np.stack([base, base + np.stack([np.zeros(npairs), gap, np.zeros(npairs)], axis=1)], axis=1).reshape(-1, 3)
    for w in (g, o):
        s = w.add_shape(orc.SPHERE, [0.5])
        for p in pos.astype(np.float32):
            w.add_body(s, tuple(map(float, p)), mass=1.0)
    for _ in range(3):
        g.step(1.0 / 60.0)
        o.set_solve_order(g.solve_order())
        o.step(1.0 / 60.0)
        np.testing.assert_array_equal(g.pairs(), o.pairs())
        assert np.abs(g.state()[:, :13] - o.state()[:, :13]).max() <= 1e-5 * max(1.0, np.abs(pos).max())
    assert g.stats()["num_contact_pairs"] == npairs - len(k[k % 3 == 1]) and g.stats()["device_status"] == 0


def test_large_pair_list_keeps_its_order():
    """More than 256k pairs: the contact pairs are the pairs with rows, ascending and complete."""
    import bgpu
    import scenes

    s = scenes.large_pile_fast(40, 40, 40, seed=2, spacing=0.99)
    w = s.build_gpu(bgpu)
    w.step(s.dt, 4)
    st = w.stats()
    assert st["num_pairs"] > (1 << 18) and st["device_status"] == 0
    keys = w.solve_order()
    assert len(keys) == st["num_contact_pairs"] == len(np.unique(keys))
    pairs = w.pairs().astype(np.uint64)
    assert np.isin(keys, (pairs[:, 0] << np.uint64(32)) | pairs[:, 1]).all()


def test_a_sleeping_world_keeps_manifolds_of_vanished_pairs():
    """A world that does not simulate does not prune: its cache is merged from both lists, and what
    wakes it later finds its warm-start impulses, as in the oracle."""
    import bgpu
    import oracle_api as orc
    import scenes

    s = scenes.falling_box_stack(3, 2, 3, seed=5)
    g, o = s.build_gpu(bgpu), s.build_oracle(orc)
    for step in range(330):
        if step == 300:  # a body far above is pushed into the sleeping stack's world
            for w in (g, o):
                w.add_body(1, (0.0, 8.0, 0.0), linvel=(0.0, -20.0, 0.0), mass=2.0)
        g.step(s.dt)
        st = g.state()
        o.set_solve_order(g.solve_order())
        o.step(s.dt)
        r = o.state()
        np.testing.assert_array_equal(st[:, 13], r[:, 13])
        assert np.abs(st[:, :13] - r[:, :13]).max() < 2e-3, step
        o.set_state(st)
    assert (g.state()[1:, 13] != 2).any()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1025])
def test_state_is_every_column_of_every_body(gpu, n):
    """A written state reads back whole: poses, velocities, activation and deactivation timer, around
    a block of the packing kernel; and again after a second, larger world state has used the staging."""
    rng = np.random.default_rng(n)
    w = gpu.World()
    w.box([0.1, 0.1, 0.1])
    for k in range(n):
        w.add_body(0, (1.0 * k, 0.0, 0.0), mass=1.0)
    s = rng.normal(size=(n, 15)).astype(np.float32)
    s[:, 3:7] /= np.linalg.norm(s[:, 3:7], axis=1, keepdims=True)
    s[:, 13] = rng.integers(1, 6, size=n)
    s[:, 14] = rng.random(n)
    w.set_state(s)
    np.testing.assert_array_equal(w.state(), s)
    np.testing.assert_array_equal(w.poses(), s[:, :7])
    w.apply_forces(np.ones((n, 3), np.float32), np.ones((n, 3), np.float32))
    np.testing.assert_array_equal(w.state(), s)


@pytest.mark.parametrize("n,leave", [(3, 1), (127, 64), (129, 128), (520, 400), (1300, 3), (1300, 700)])
def test_old_manifolds_are_found(gpu, n, leave):
    """Boxes on one static box settle, then all but a few leave at once: the pairs of a block look for
    their manifolds among few old keys, among more than a block stages, and where none is left. In
    lockstep with the oracle, whose impulses start from the same manifolds."""
    import oracle_api as orc
    from test_gpu_lockstep import lockstep

    side = int(np.ceil(np.sqrt(n)))
    w, o = gpu.World(), orc.OracleWorld("f32")
    for x in (w, o):
        assert [x.box([1.5 * side, 0.5, 1.5 * side]), x.box([0.5, 0.5, 0.5])] == [0, 1]
        x.add_body(0, (0.0, -0.5, 0.0), mass=0.0)
        for k in range(n):
            x.add_body(1, (1.25 * (k % side - side / 2), 0.499, 1.25 * (k // side - side / 2)), mass=1.0)
    lockstep(w, o, 1.0 / 60.0, 3, "settle")
    s = w.state()
    stay = np.zeros(n + 1, bool)
    stay[0] = True
    stay[1 + np.linspace(0, n - 1, leave).astype(int)] = True
    s[~stay, 1] += 50.0
    w.set_state(s)
    lockstep(w, o, 1.0 / 60.0, 2, "after")
    assert len(w.pairs()) == leave
