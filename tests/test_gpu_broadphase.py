"""The pair list on both sides of the all-pairs limit (12,288 proxies) and at the edges of its tiles,
bit for bit against the all-pairs definition: bounded proxies, planes among them, dense clusters
with more partners than a stash holds, identical boxes, boxes that touch in a face."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path[:0] = [os.path.join(ROOT, "bullet-physics_b200"), os.path.join(ROOT, "tests")]


def _expected(a):
    out = []
    for i in range(len(a)):
        hit = np.all((a[i, 0:3] <= a[i + 1:, 3:6]) & (a[i + 1:, 0:3] <= a[i, 3:6]), axis=1)
        j = np.flatnonzero(hit) + i + 1
        out.append(np.stack([np.full(len(j), i), j], axis=1))
    return np.concatenate(out).astype(np.uint32)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 65, 127, 129, 256, 257, 1000, 4097, 12287, 12288, 12289, 14000])
def test_pairs_equal_the_definition(n):
    import bgpu

    rng = np.random.default_rng(n)
    side = max(2.0, (n * 0.5) ** (1.0 / 3.0) * 1.6)
    c = rng.uniform(0.0, side, size=(n, 3))
    h = rng.uniform(0.2, 0.6, size=(n, 3))
    c[: n // 10] = rng.uniform(0.0, 1.2, size=(n // 10, 3)) if n < 3000 else c[: n // 10]
    c[n // 2: n // 2 + min(80, n // 4)] = c[n // 2]  # a cluster of more than 32 partners each
    h[n // 3: n // 3 + min(50, n // 5)] = h[n // 3]
    c[n // 3: n // 3 + min(50, n // 5)] = c[n // 3]  # identical boxes
    a = np.concatenate([c - h, c + h], axis=1).astype(np.float32)
    k = n // 4
    if n > 20:
        a[k + 1, 0:3], a[k + 1, 3:6] = a[k, 0:3], a[k, 3:6]
        a[k + 1, [0, 3]] = a[k, 3], a[k, 3] + np.float32(1.0)  # touches in a face
        a[[5, n // 2 + 1, n - 1]] = [-1e30, -1e30, -1e30, 1e30, 1e30, 1e30]  # unbounded
    np.testing.assert_array_equal(bgpu.broadphase_pairs(a), _expected(a))


@pytest.mark.parametrize("n", [12100, 12400])
def test_a_world_that_grows_across_the_limit_and_sleeps(n):
    """Two worlds stepped by both paths from the same bodies: pairs as by the definition, and a body
    added later takes a world from the all-pairs pass to the tree."""
    import bgpu

    rng = np.random.default_rng(3)
    w = bgpu.World(num_iterations=4)
    plane, sph = w.plane([0, 1, 0], 0.0), w.sphere(0.5)
    w.add_body(plane, (0, 0, 0), mass=0.0)
    pos = rng.uniform(0.0, 30.0, size=(n, 3)) + [0, 1, 0]
    w.add_bodies_array(np.full(n, sph), pos, np.tile([0, 0, 0, 1], (n, 1)), mass=np.ones(n))
    other = w.plane([1, 0, 0], -40.0)
    for step in range(4):
        if step == 2:
            w.add_body(other, (0, 0, 0), mass=0.0)
            w.add_bodies_array(np.full(300, sph), rng.uniform(0, 30, size=(300, 3)), np.tile([0, 0, 0, 1], (300, 1)),
                               mass=np.ones(300))
        before = w.state()
        w.step(1.0 / 60.0)
        # predicted pose and padded box of this step's velocities
        v = before[:, 7:10] + np.float32([0, -9.81, 0]) * np.float32(1 / 60)
        p = before[:, 0:3] + v * np.float32(1 / 60)
        got = w.pairs()
        lo, hi = p - 0.52, p + 0.52
        isp = np.zeros(len(p), bool)
        isp[0] = True
        if step >= 2:
            isp[n + 1] = True
        lo[isp], hi[isp] = -1e30, 1e30
        exp = _expected(np.concatenate([lo, hi], axis=1).astype(np.float32))
        key = lambda q: q[:, 0].astype(np.uint64) << np.uint64(32) | q[:, 1].astype(np.uint64)
        g, e = key(got), key(exp)
        assert (np.diff(g.astype(np.int64)) > 0).all()
        # rounding of the box edges may differ by an ulp: all but touching boxes agree
        assert len(np.setxor1d(g, e)) <= 3
        assert w.stats()["device_status"] == 0


@pytest.mark.parametrize("n", [2, 3, 511, 512, 513, 1024, 1025, 3000])
def test_tree_at_the_edges_of_a_refit_block(n):
    """The allocation-free entry takes the tree at every size: one block of leaves, its remainders, a
    last block of one leaf, and a third of the boxes identical (equal keys, a deep subtree across blocks)."""
    import ctypes

    import torch

    import bgpu
    from test_zz_no_alloc import _entry

    rng = np.random.default_rng(n)
    c = rng.uniform(0.0, max(2.0, n ** (1.0 / 3.0)), size=(n, 3))
    h = rng.uniform(0.1, 0.5, size=(n, 3))
    c[n // 3: n // 3 + min(n // 3, 600)] = c[n // 3]
    h[n // 3: n // 3 + min(n // 3, 600)] = 0.01
    a = np.concatenate([c - h, c + h], axis=1).astype(np.float32)
    want = _expected(a)
    dev = torch.from_numpy(a).cuda()
    out = torch.full((len(want) + 8, 2), -1, dtype=torch.int32, device="cuda")
    got = ctypes.c_uint64(0)
    torch.cuda.synchronize()
    assert _entry(bgpu)(dev.data_ptr(), n, out.data_ptr(), len(want) + 8, ctypes.byref(got), None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out[: got.value].cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("meshes", [1, 4680, 4682, 9500])
def test_many_proxies_outside_the_tree(meshes):
    """Meshes are kept out of the tree, 14 tiles of 1,024 proxies each: 4,681 of them take a launch, more take
    two and three. Small meshes among spheres, a few meshes under a crowd, against the oracle's
    brute force."""
    import bgpu
    import oracle_api as orc

    n = 14000
    rng = np.random.default_rng(meshes)
    side = (n * 0.3) ** (1.0 / 3.0) * 1.5
    pos = rng.uniform(0.0, side, size=(n, 3))
    kind = np.full(n, 1)
    kind[rng.permutation(n)[:meshes]] = 0
    big = np.flatnonzero(kind == 0)[::997]
    worlds = []
    for x in (bgpu.World(gravity=(0.0, 0.0, 0.0), num_iterations=1), orc.OracleWorld("f32")):
        x.set_gravity((0.0, 0.0, 0.0))
        tri = [[-0.3, 0.0, -0.3], [0.3, 0.1, -0.3], [0.0, 0.2, 0.3]]
        assert [x.mesh(np.asarray(tri, np.float32), [[0, 2, 1]]), x.sphere(0.25),
                x.mesh(20.0 * np.asarray(tri, np.float32), [[0, 2, 1]])] == [0, 1, 2]
        k = kind.copy()
        k[big] = 2
        for i in range(n):
            x.add_body(int(k[i]), tuple(pos[i]), mass=1.0 if k[i] == 1 else 0.0)
        worlds.append(x)
    w, o = worlds
    o.set_brute_force(True)
    w.step(1.0 / 240.0)
    o.step(1.0 / 240.0)
    np.testing.assert_array_equal(w.pairs(), o.pairs())
    assert np.bincount(w.pairs()[:, 0]).max() > 32
