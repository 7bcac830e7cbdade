"""Obstacle normals of moving obstacles (through the boxes they grow) against the CPU oracle, bit for
bit: poles with rings shorter and longer than a round of entries, vertex counts around a warp."""
import numpy as np
import pytest

from tests.helpers import bits, make_pair
from xrtailor_gb300 import scenes
from xrtailor_gb300.solver import Mesh

pytestmark = pytest.mark.gpu


def _cone(ring, pole_last):
    t = np.arange(ring) * 2 * np.pi / ring
    rim = np.stack([0.5 + 0.4 * np.cos(t), np.full(ring, 0.05), 0.5 + 0.4 * np.sin(t)], 1)
    rim[:, 1] += np.random.default_rng(ring).normal(0, 0.01, ring)
    p = np.vstack([rim, [[0.5, 0.2, 0.5]]] if pole_last else [[[0.5, 0.2, 0.5]], rim])
    first, pole = (0, ring) if pole_last else (1, 0)
    k = np.arange(ring)
    tri = np.stack([np.full(ring, pole), first + (k + 1) % ring, first + k], 1)
    return Mesh(p.astype(np.float32), tri.astype(np.uint32))


@pytest.mark.parametrize("pole_last", [False, True])
@pytest.mark.parametrize("ring", [3, 31, 64, 192, 500])
def test_cone_matches_oracle(xrt, ring, pole_last):
    cloth = scenes.grid_cloth(12, 1.0, origin=(0.0, 0.25, 0.0), jitter=1e-3, seed=3)
    obstacle = _cone(ring, pole_last)
    p = scenes._params(num_substeps=2, num_iterations=2, num_collision_passes=2, solve_bending=0,
                       enable_self_collision=0)
    g, o = make_pair(p, [cloth], [obstacle])
    for f in range(3):
        target = obstacle.positions + np.float32(0.01 * (f + 1))
        for s in (g, o):
            s.set_obstacle_targets(target)
            s.step()
        a, b = g.export_obstacle_bvh(), o.export_obstacle_bvh()
        np.testing.assert_array_equal(bits(a["aabbs"]), bits(b["aabbs"]))
        np.testing.assert_array_equal(bits(g.host_positions()), bits(o.host_positions()))
