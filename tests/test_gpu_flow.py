"""The chunked PGS kernel at the edges of its deal, against the team kernel, bit for bit.

Both solve the groups in (sweep, colour, pair) order, so every state must be identical: a warp with
one item a sweep (few groups a chunk), several rounds of a colour, groups of 1 to 4 rows in one
warp, split groups of a deep initial overlap, kinematic bodies, no velocity sweep and a single one.
BGPU_PGS=team selects the team kernel (read once per process), hence the child processes.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
sys.path[:0] = [sys.argv[1] + "/bullet-physics_b200"]
import numpy as np
import bgpu, scenes
kind, iters, steps = sys.argv[2], int(sys.argv[3]), int(sys.argv[4])
if kind == "boxes":        # 1,050 bodies: the smallest worlds the kernel takes, a few groups a chunk
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
