"""The one-walk tree build and refit (csrc/lbvh_dev.cuh tree_up) and the one-cluster front end of
small trees against the CPU oracle, bit for bit, at the edges of their blocks and rounds."""
import numpy as np
import pytest

from tests.helpers import prim_soup
from tests.test_lbvh_gpu import _pair, _same_tree

pytestmark = pytest.mark.gpu


def _prims(kind, n):
    p = prim_soup(n, seed=n)
    if kind == "line":       # one long chain of cells: an unbalanced tree, walks across many blocks
        p = (np.linspace(0, 1, n, dtype=np.float32)[:, None] ** 8 + p * 1e-2).astype(np.float32)
    elif kind == "copies":   # runs of equal codes, some longer than a block
        p = p[np.sort(np.random.default_rng(n).integers(0, max(n // 300, 1), n))]
    return np.ascontiguousarray(p)


# 256-leaf blocks, the sort's rounds of 8,192, the last one-cluster size (16,384) and the first above
@pytest.mark.parametrize("n", [2, 9, 255, 257, 1023, 8192, 8193, 16383, 16384, 16385, 33000])
@pytest.mark.parametrize("kind", ["soup", "line", "copies"])
def test_build_and_refit_match_oracle(xrt, kind, n):
    p = _prims(kind, n)
    g, o = _pair(p)
    _same_tree(g, o)
    rng = np.random.default_rng(n + 1)
    for _ in range(2):
        moved = (p + rng.normal(0, 0.02, p.shape)).astype(np.float32)
        g.refit(moved)
        o.refit(moved)
        _same_tree(g, o)


def test_rebuilds_of_changing_size_share_a_handle(xrt):
    from oracle.oracle import OracleLbvh
    from xrtailor_gb300 import Lbvh
    g = Lbvh()
    for n in (40000, 300, 9000, 1, 70000, 257):
        p = prim_soup(n, seed=n)
        o = OracleLbvh()
        g.build(p)
        o.build(p, None, 0.0)
        _same_tree(g, o)
        g.refit(p + np.float32(0.25))
        o.refit(p + np.float32(0.25))
        _same_tree(g, o)
