"""LRA + VF + EE solve against the CPU oracle, bit for bit: fewer and more slots than are read ahead
of the wait, and more vertices than the lists are read ahead for (97,280)."""
import numpy as np
import pytest

from tests.helpers import bits, make_pair
from xrtailor_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 313])  # 400 and 97,969 vertices
@pytest.mark.parametrize("slots", [1, 2, 5])
def test_frames_match_oracle(xrt, n, slots):
    cloth = scenes.grid_cloth(n, 1.0, origin=(0.0, 0.305, 0.0), jitter=1e-4, seed=slots)
    pins = np.array([0, n - 1, n * n - 1, n * n - n, n // 2], np.uint32)[:slots]
    cloth.fixed_indices = cloth.attached_indices = pins
    obstacle = scenes.icosphere(3, 0.3, center=(0.5, 0.0, 0.5))
    p = scenes._params(num_substeps=2, num_iterations=2, num_collision_passes=2, solve_bending=0,
                       enable_self_collision=0)
    g, o = make_pair(p, [cloth], [obstacle])
    hits = 0
    for _ in range(3):
        g.step()
        o.step()
        hits += (g.export_contacts()["vf_index"] >= 0).sum()
    assert hits > 0
    a, b = g.host_positions(), o.host_positions()
    assert np.isfinite(b).all()
    np.testing.assert_array_equal(bits(a), bits(b))
