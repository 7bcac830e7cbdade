"""Boxes of trees whose merge crosses blocks (more than 16,384 leaves, or a forest), built and refitted
again and again in the same memory with quite different positions, against the CPU oracle: a node that
a merge reads before it is written would show as the box of the round before."""
import numpy as np
import pytest

from tests.helpers import bits, prim_soup
from tests.test_lbvh_gpu import _same_tree

pytestmark = pytest.mark.gpu


def _round(n, k):
    """Round k: everything far from where the other rounds have it."""
    p = prim_soup(n, seed=100 + k).reshape(n, 3, 3)
    far = np.float32(50.0) * np.array([np.cos(k), np.sin(k), (-1) ** k], np.float32)
    return np.ascontiguousarray((p * np.float32(1 + k) + far).reshape(n, 9))


@pytest.mark.parametrize("n", [16385, 120000, 400000])
def test_large_tree_rounds_match_oracle(xrt, n):
    from oracle.oracle import OracleLbvh
    from xrtailor_gb300 import Lbvh
    g, o = Lbvh(), OracleLbvh()
    for k in range(4):
        for s in (g, o):
            s.build(_round(n, k), None, 0.0)
        _same_tree(g, o)
        for j in (k + 1, k + 2):
            for s in (g, o):
                s.refit(_round(n, j))
            _same_tree(g, o)


def test_forest_rounds_match_single_trees(xrt):
    """Bodies of 20 to 20,480 triangles share one forest; each must have the boxes of its own tree."""
    from xrtailor_gb300 import ClothSolver, scenes
    p = scenes._params(num_substeps=2, num_iterations=2, num_collision_passes=2, solve_bending=0,
                       enable_self_collision=0, update_obstacle_animation=1)
    cloth = scenes.grid_cloth(4, 1.0, origin=(0.0, 3.0, 0.0), jitter=1e-3, seed=1)
    bodies = [scenes.icosphere(k, 0.3, center=(0.5, 0.0, 0.5)) for k in (5, 0, 3, 4, 5, 1, 5)]
    batch = ClothSolver(p)
    for b in bodies:
        batch.add_instance(cloth, b)
    batch.start()
    single = {}
    for k, b in enumerate(bodies):
        if len(b.positions) in single:
            continue
        s = ClothSolver(p)
        s.add_cloth(cloth)
        s.add_obstacle(b)
        s.start()
        single[len(b.positions)] = s
    for k in range(8):
        def moved(b):
            c = np.array([np.cos(2.1 * k), 0.3 * np.sin(k), np.sin(1.7 * k)], np.float32)
            return (b.positions * np.float32(1 + 0.5 * (k % 3)) + np.float32(20) * c).astype(np.float32)
        for b in bodies:
            single[len(b.positions)].set_obstacle_targets(moved(b))
        batch.set_obstacle_targets(np.concatenate([moved(b) for b in bodies]))
        for s in [batch, *single.values()]:
            s.step()
        trees = {n: s.export_obstacle_bvh() for n, s in single.items()}
        f = batch.export_obstacle_bvh()
        node = 0
        for b in bodies:
            t = trees[len(b.positions)]
            m = len(t["aabbs"])
            np.testing.assert_array_equal(f["nodes"][node:node + m], t["nodes"])
            np.testing.assert_array_equal(bits(f["aabbs"][node:node + m]), bits(t["aabbs"]))
            node += m
        assert node == len(f["aabbs"])


def test_ccd_refit_rounds_match_oracle(xrt):
    """The obstacle's boxes grow by its motion, refit after refit, each further out than the one before."""
    from tests.helpers import make_pair
    from xrtailor_gb300 import scenes
    body = scenes.icosphere(5, 0.3, center=(0.5, 0.0, 0.5))  # 20,480 triangles
    cloth = scenes.grid_cloth(4, 1.0, origin=(0.0, 3.0, 0.0), jitter=1e-3, seed=1)
    p = scenes._params(num_substeps=1, num_iterations=1, num_collision_passes=1, solve_bending=0,
                       enable_self_collision=0)
    g, o = make_pair(p, [cloth], [body])
    rng = np.random.default_rng(3)
    for k in range(8):
        far = rng.normal(0, 5.0 * (k + 1), 3).astype(np.float32)
        target = (body.positions * np.float32(1 + k) + far).astype(np.float32)
        for s in (g, o):
            s.set_obstacle_targets(target)
            s.obstacle_bvh_update_ccd()
        a, b = g.export_obstacle_bvh(), o.export_obstacle_bvh()
        np.testing.assert_array_equal(a["nodes"], b["nodes"])
        np.testing.assert_array_equal(bits(a["aabbs"]), bits(b["aabbs"]))
