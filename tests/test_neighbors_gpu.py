"""Neighbor lists against the CPU oracle, in list order: clumps of more entries than a warp tests at
once, lists from empty to the cap, in both kernels (a warp per vertex; a lane per vertex above
243,200 vertices)."""
import numpy as np
import pytest

from oracle.oracle import OracleSolver
from xrtailor_gb300 import ClothSolver, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 500])  # 4, 1,089 and 250,000 vertices
@pytest.mark.parametrize("cap, cell", [(64, 1.5), (3, 1.5), (64, 3.0)])
def test_lists_match_oracle(xrt, n, cap, cell):
    rng = np.random.default_rng(n + cap)
    d = 0.02
    cloth = scenes.grid_cloth(n, 1.0, jitter=0.0, seed=2)
    x = np.empty((n * n, 3), np.float32)
    for k, side in enumerate((30.0, 12.0, 8.0, 5.0)):
        part = np.arange(k, n * n, 4)
        x[part] = rng.uniform(0, 2 * side * d * (len(part) / 272.0) ** (1 / 3), (len(part), 3))
        x[part] += 100.0 * k
    cloth.positions = x
    p = scenes._params(num_substeps=1, num_iterations=1, num_collision_passes=1, solve_bending=0,
                       stretch_compliance=1e-2, max_neighbor_size=cap, hash_cell_size=cell)
    half = np.diag([0.5, 0.5, 0.5, 1.0]).astype(np.float32)
    g, o = ClothSolver(p), OracleSolver(p)
    for s in (g, o):
        s.add_cloth(cloth, half, particle_diameter=d)
    g.start()
    o.set_coloring(0, g.coloring(0))
    o.set_coloring(1, g.coloring(1))
    o.start()
    g.step()
    o.step()
    a = g.export_neighbors().reshape(-1, n * n)
    b = o.export_neighbors().reshape(-1, n * n)

    def cut(lists):  # what follows a list's end is left over from before
        ended = np.cumsum(lists >= n * n, axis=0) > 0
        return np.where(ended, n * n, lists)

    np.testing.assert_array_equal(cut(a), cut(b))
