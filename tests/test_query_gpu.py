"""Tree queries against the CPU oracle, candidates in walk order: none, few, more than the cap and more
nodes at once than a warp's list holds, in both kernels (a warp per query; a lane per query above
20,000 queries)."""
import numpy as np
import pytest

from tests.helpers import prim_soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 300, 6000])
@pytest.mark.parametrize("nq", [1, 130, 20001])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_candidates_match_oracle(xrt, n, nq, kind):
    from oracle.oracle import OracleLbvh
    from xrtailor_gb300 import Lbvh
    prims = prim_soup(n, seed=n)
    g, o = Lbvh(), OracleLbvh()
    g.build(prims, None, 0.02)
    o.build(prims, None, 0.02)
    rng = np.random.default_rng(nq + kind)
    a = rng.uniform(-1.2, 1.2, (nq, 3))
    if kind == 0:
        q = a
    elif kind == 1:
        q = np.concatenate([a, a + rng.normal(0, 0.3, (nq, 3))], 1)
    else:
        half = rng.choice([0.0, 0.05, 0.3, 0.8, 3.0], (nq, 1), p=[0.2, 0.4, 0.2, 0.1, 0.1])
        q = np.concatenate([a - half, a + half], 1)
    q = q.astype(np.float32)
    cg, kg = g.query(kind, q)
    co, ko = o.query(kind, q)
    np.testing.assert_array_equal(cg, co)
    live = np.arange(kg.shape[1])[None, :] < cg[:, None]
    np.testing.assert_array_equal(np.where(live, kg, 0), np.where(live, ko, 0))
