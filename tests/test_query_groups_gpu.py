"""Tree queries by 32 lanes (up to 3,000 queries) and by 8 lanes (up to 20,000) against the CPU oracle,
candidates in walk order, at the edges between the kernels; and walks whose nodes all overlap while few
leaves do, which fill the stack of 8 lanes until entries are taken singly."""
import numpy as np
import pytest

from tests.helpers import prim_soup

pytestmark = pytest.mark.gpu


def _same(cg, kg, co, ko):
    np.testing.assert_array_equal(cg, co)
    live = np.arange(kg.shape[1])[None, :] < cg[:, None]
    np.testing.assert_array_equal(np.where(live, kg, 0), np.where(live, ko, 0))


@pytest.mark.parametrize("n", [1, 2, 300, 40000])
@pytest.mark.parametrize("nq", [3000, 3001, 3007, 20000])
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
    _same(*g.query(kind, q), *o.query(kind, q))


def _spine(depth, bushy):
    """Keys (bit strings) of a tree whose left spine is `depth` long and whose right children are
    balanced trees of up to 2^bushy leaves."""
    keys = ["0" * depth]
    for j in range(depth):
        b = min(depth - 1 - j, bushy)
        keys += ["0" * j + "1" + (format(k, f"0{b}b") if b else "") for k in range(1 << b)]
    return sorted(k.ljust(depth, "0") for k in keys)


def _full_tree(hits):
    """Triangles with those Morton codes whose inner nodes all hold the point q while only `hits` leaves
    do: a leaf is wide in x and narrow in y or the other way round, in turn along the codes."""
    keys = _spine(24, 4)
    q = np.array([0.375, 0.375, 0.375])
    rng = np.random.default_rng(hits)
    both = set(rng.choice(len(keys), hits, replace=False).tolist())
    tri = [np.zeros((3, 3)) + [[0, 0, 0], [2e-5, 2e-5, 2e-5], [0, 2e-5, 0]],
           np.ones((3, 3)) - [[0, 0, 0], [2e-5, 2e-5, 2e-5], [0, 2e-5, 0]]]  # the root is [0, 1]^3
    for i, key in enumerate(keys):
        code = "000" "111" + key           # x, y and z in [0.25, 0.5)
        cell = np.array([int(code[a::3], 2) for a in range(3)])
        c = (cell + 0.5) / 1024
        half = np.abs(c - q) + 0.01
        if i not in both:
            half[i % 2] = 1e-5
        lo, hi = c - half, c + half
        tri.append(np.array([lo, hi, [lo[0], hi[1], lo[2]]]))
    tri = np.array(tri)[rng.permutation(len(tri))]
    return tri.astype(np.float32).reshape(-1, 9), q.astype(np.float32)


@pytest.mark.parametrize("nq", [1, 70, 3001])
@pytest.mark.parametrize("hits", [0, 5, 300])
@pytest.mark.parametrize("kind", [0, 2])
def test_full_stacks(xrt, nq, hits, kind):
    from oracle.oracle import OracleLbvh
    from xrtailor_gb300 import Lbvh
    prims, q = _full_tree(hits)
    g, o = Lbvh(), OracleLbvh()
    g.build(prims)
    o.build(prims, None, 0.0)
    qs = np.tile(q if kind == 0 else np.concatenate([q, q]), (nq, 1)).astype(np.float32)
    co, ko = o.query(kind, qs)
    assert (co == min(hits, 256)).all()
    _same(*g.query(kind, qs), co, ko)
