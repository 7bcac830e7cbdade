"""Tile launches of more tiles than the GPU holds at once: small tiles with whole records, large ones
with records streamed by local color.  Copies of one cloth in a batch step as the cloth alone, whose
launches are resident."""
import numpy as np
import pytest

from tests.helpers import bits
from xrtailor_gb300 import ClothSolver, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile, copies", [(32, 16), (64, 24), (512, 90)])
def test_copies_match_one(xrt, tile, copies):
    cloth = scenes.grid_cloth(100, 1.0, jitter=1e-3, seed=7)
    cloth.fixed_indices = scenes.two_corner_pins(100)
    p = scenes._params(num_substeps=2, num_iterations=3, num_collision_passes=1,
                       stretch_compliance=1e-8, bend_compliance=1e-6, enable_self_collision=0)

    def make(count):
        s = ClothSolver(p)
        s.set_tile_vertices(tile)
        for _ in range(count):
            s.add_instance(cloth)
        s.start()
        return s

    one, many = make(1), make(copies)
    colors = many.sizes().num_stretch_tile_colors
    assert copies * (10000 // tile) / colors > 4 * 152 or tile == 512  # 256-thread blocks: four an SM
    assert copies * (10000 // tile) / colors > 2 * 152                 # 512-thread blocks: two
    for _ in range(3):
        one.step()
        many.step()
    x = one.host_positions()
    assert np.isfinite(x).all() and np.abs(x - cloth.positions).max() > 1e-3
    np.testing.assert_array_equal(bits(many.host_positions().reshape(copies, -1)),
                                  np.tile(bits(x).reshape(1, -1), (copies, 1)))
