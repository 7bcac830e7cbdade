"""Particle push-out of piled vertices against the CPU oracle, bit for bit: lists from empty to
the cap or beyond two batches of slots, pairs of two pinned vertices, without friction, in both kernels (four lanes per vertex; a queue
of pairs per warp above 109,440 vertices)."""
import numpy as np
import pytest

from oracle.oracle import OracleSolver
from tests.helpers import bits
from xrtailor_gb300 import ClothSolver, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 331])  # 1,089 and 109,561 vertices: a ragged last warp in each
@pytest.mark.parametrize("cap, mu", [(64, 0.1), (5, 0.1), (8, 0.0), (9, 0.1), (17, 0.5)])
def test_pile_matches_oracle(xrt, n, cap, mu):
    rng = np.random.default_rng(n + cap)
    d = 0.02 if n == 33 else 0.004
    cloth = scenes.grid_cloth(n, 1.0, jitter=0.0, seed=2)
    # clumps of different density, a quarter of the vertices each; the state is the mesh at half its
    # size, so every edge pushes its ends apart
    x = np.empty((n * n, 3), np.float32)
    for k, side in enumerate((30.0, 12.0, 8.0, 5.0)):
        part = np.arange(k, n * n, 4)
        scale = 2 * side * d * (len(part) / 272.0) ** (1 / 3)
        x[part] = rng.uniform(0, scale, (len(part), 3)) + 10.0 * k
    cloth.positions = x
    cloth.fixed_indices = np.arange(0, n * n, 7, dtype=np.uint32)
    p = scenes._params(num_substeps=2, num_iterations=3, num_collision_passes=1, solve_bending=0,
                       stretch_compliance=1e-2, max_neighbor_size=cap, friction=mu,
                       inter_leaved_hash=1, hash_cell_size=2.5)
    half = np.diag([0.5, 0.5, 0.5, 1.0]).astype(np.float32)
    g, o = ClothSolver(p), OracleSolver(p)
    for s in (g, o):
        s.add_cloth(cloth, half, particle_diameter=d)
    g.start()
    o.set_coloring(0, g.coloring(0))
    o.set_coloring(1, g.coloring(1))
    o.start()
    for _ in range(2):
        g.step()
        o.step()
    a, b = g.host_positions(), o.host_positions()
    assert np.isfinite(b).all()
    np.testing.assert_array_equal(bits(a), bits(b))
    lists = g.export_neighbors().reshape(-1, n * n)
    ends = lists >= n * n
    length = np.where(ends.any(0), ends.argmax(0), cap)
    assert length.min() == 0 and length.max() >= min(cap, 17)  # empty, full or three batches long
