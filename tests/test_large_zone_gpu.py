"""A zone of more impacts than the 16,384 threads of the widest cluster: the kernel that keeps an element
per thread does not take it, the one that loops over chunks does."""
import numpy as np
import pytest

from tests.helpers import bits, make_pair
from xrtailor_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_zone_beyond_the_widest_cluster_matches_oracle(xrt):
    n = 136
    sheet = scenes.grid_cloth(n, 1.0, origin=(0.0, 0.5, 0.0), jitter=1.6e-2 / n, seed=3)
    floor = scenes.grid_cloth(n, 1.0, origin=(0.8 / n, 0.5 - 0.8 / n, 0.8 / n), jitter=1.6e-2 / n, seed=4)
    p = scenes._params(num_substeps=2, num_iterations=3, solve_bending=0, num_collision_passes=2,
                       enable_self_collision=0)
    g, o = make_pair(p, [sheet], [floor])
    pred = o.host_positions()
    pred[:, 1] -= np.float32(0.96 / n)
    g.set_predicted(pred)
    o.set_predicted(pred)
    sg = g.collision_step(launch_shapes=True)
    so = o.collision_step()
    shapes = sg.pop("wide_solves")
    # one zone holds all impacts, so its last solve has more of them than the cluster has threads
    assert sg == so and sg["success"] == 1 and sg["zones"] == 1 and sg["impacts"] > 16384, (sg, so)
    assert shapes[1] > 0, shapes
    np.testing.assert_array_equal(bits(g.predicted()), bits(o.predicted()))
