"""Obstacles of more vertices than one wave of spread fans (77,824): a lane per vertex without poles,
spread fans with a long ring, against the CPU oracle, bit for bit, through the boxes they grow."""
import numpy as np
import pytest

from tests.helpers import bits, make_pair
from tests.test_fan_gpu import _cone
from xrtailor_gb300 import scenes
from xrtailor_gb300.solver import Mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ring", [None, 500])
def test_large_obstacle_matches_oracle(xrt, ring):
    n = 280  # 78,400 vertices
    m = scenes.rect_cloth(n, n, 3.0, 3.0, origin=(-1.0, -0.1, -1.0), jitter=1e-3, seed=4)
    p, t = m.positions, m.triangles
    if ring:
        c = _cone(ring, True)
        p, t = np.concatenate([p, c.positions]), np.concatenate([t, c.triangles + len(p)])
    p = p.copy()
    p[:, 1] += 0.02 * np.sin(9 * p[:, 0]) * np.cos(7 * p[:, 2])
    obstacle = Mesh(p.astype(np.float32), t.astype(np.uint32))
    cloth = scenes.grid_cloth(12, 1.0, origin=(0.0, 0.25, 0.0), jitter=1e-3, seed=3)
    q = scenes._params(num_substeps=2, num_iterations=2, num_collision_passes=2, solve_bending=0,
                       enable_self_collision=0)
    g, o = make_pair(q, [cloth], [obstacle])
    for f in range(3):
        wave = obstacle.positions.copy()
        wave[:, 1] += np.float32(0.01 * (f + 1)) * np.sin(5 * wave[:, 0] + f).astype(np.float32)
        for s in (g, o):
            s.set_obstacle_targets(wave)
            s.step()
        a, b = g.export_obstacle_bvh(), o.export_obstacle_bvh()
        np.testing.assert_array_equal(bits(a["aabbs"]), bits(b["aabbs"]))
        np.testing.assert_array_equal(bits(g.host_positions()), bits(o.host_positions()))
