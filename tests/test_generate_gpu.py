"""Contact generation (nearest point, ray hit, nearest owned edge) against the CPU oracle, bit for
bit, contacts and frames: trees of one leaf and of several hundred, walks that end at the root and
walks that meet more leaves than the cap, query counts around a warp and around its refills."""
import numpy as np
import pytest

from tests.helpers import bits, make_pair
from xrtailor_gb300 import scenes
from xrtailor_gb300.solver import Mesh

pytestmark = pytest.mark.gpu


def _one_triangle():
    p = np.array([[-2, 0.2, -2], [3, 0.25, -2], [0.5, 0.15, 4]], np.float32)
    return Mesh(p, np.array([[0, 2, 1]], np.uint32))


OBSTACLES = {
    "triangle": _one_triangle,
    "sphere": lambda: scenes.icosphere(3, 0.3, center=(0.5, 0.1, 0.5)),
    "far": lambda: scenes.icosphere(1, 0.3, center=(50.0, 0.0, 0.5)),
}


@pytest.mark.parametrize("n", [3, 6, 33])  # 9, 36 and 1,089 vertices
@pytest.mark.parametrize("obstacle, tolerance", [("triangle", 1e-2), ("sphere", 1e-3),
                                                 ("sphere", 0.15), ("sphere", 5.0), ("far", 1e-2)])
def test_frames_match_oracle(xrt, n, obstacle, tolerance):
    cloth = scenes.grid_cloth(n, 1.0, origin=(0.0, 0.3, 0.0), jitter=1e-3, seed=n)
    p = scenes._params(num_substeps=2, num_iterations=2, num_collision_passes=2,
                       enable_self_collision=0, solve_bending=0, bvh_tolerance=tolerance)
    g, o = make_pair(p, [cloth], [OBSTACLES[obstacle]()])
    hits = 0
    for _ in range(6):
        g.step()
        o.step()
        cg, co = g.export_contacts(), o.export_contacts()
        for k in ("vf_index", "rt_index"):
            np.testing.assert_array_equal(cg[k], co[k])
        for k in ("vf_qs", "rt_qc", "ee"):
            np.testing.assert_array_equal(bits(cg[k]), bits(co[k]))
        hits += (cg["vf_index"] >= 0).sum()
    assert hits > 0 or tolerance < 5.0
    a, b = g.host_positions(), o.host_positions()
    assert np.isfinite(b).all()
    np.testing.assert_array_equal(bits(a), bits(b))
